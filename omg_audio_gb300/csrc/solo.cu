// The tracer for launches of few rays: one warp per ray.
//
// What bounds such a launch is one ray's chain of segments, each a chain of
// dependent loads and instructions: a lane walking the binary tree alone takes
// some 25,000 cycles a segment on a 50k-primitive scene (20 node steps of 75
// instructions and an L2 trip each, the leaves, a dozen panel groups), and the
// other lanes of its warp add only divergence. Here the 32 lanes work on one
// ray's segment together:
//   - the walk goes over many nodes and leaves at once (solo_walk.cuh);
//   - the panels are tested one a lane;
//   - the shading pass runs uniformly, every lane the same values.
#include "shade_common.cuh"
#include "solo_walk.cuh"

namespace omg {

namespace {

constexpr uint32_t kSoloThreads = 64;
// Blocks a multiprocessor: 24 warps at 80 registers for the walk (4096 rays on the
// 40-room world, first-found and near-tie rule: 748 and 615 us a call, 766 and 668
// at 14, 817 and 669 at 16, 796 and 675 at 11), 28 at 72 for launches of small
// meshes alone (ALL), which carry no walk (4096 rays in a 12-triangle room 393 us,
// 406 at 16, 466 at 12; 474 with the walk beside it).
constexpr uint32_t kSoloBlocks = 12;
constexpr uint32_t kAllBlocks = 14;

// panels_hit (shade_common.cuh), one panel a lane: the reference's slab entry
// test, the nearest entry, the lowest original index among equal ones.
__device__ __forceinline__ bool solo_panels(const DJob& J, const DPanel* __restrict__ panels,
                                            const DMat* __restrict__ job_mats, float px, float py, float pz, float dx,
                                            float dy, float dz, bool have, Hit& h) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const float p[3] = {px, py, pz}, d[3] = {dx, dy, dz};
  float bt = FLT_MAX;
  uint32_t b_orig = 0xFFFFFFFFu, b_mat = 0;
  int b_axis = 0;
  for (uint32_t i = lane; i < J.n_panels; i += 32u) {
    const DPanel& pn = panels[J.panel_off + i];
    float t0 = 0.0f, t1 = FLT_MAX;
    int axis = 3;
    bool miss = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float da = d[a], pa = p[a], lo = pn.mn[a], hi = pn.mx[a];
      if (fabsf(da) < 1e-9f) {
        if (pa < lo || pa > hi) miss = true;
      } else {
        float ta = (lo - pa) / da, tb = (hi - pa) / da;
        if (ta > tb) { const float tmp = ta; ta = tb; tb = tmp; }
        if (ta > t0) { t0 = ta; axis = a; }
        t1 = fminf(t1, tb);
        if (t0 > t1) miss = true;
      }
    }
    if (!miss && t0 > 1e-4f && t0 < FLT_MAX && axis < 3 && (t0 < bt || (t0 == bt && pn.orig < b_orig))) {
      bt = t0;
      b_orig = pn.orig;
      b_mat = pn.mat;
      b_axis = axis;
    }
  }
  __syncwarp();
  const float tm = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(bt)));
  if (tm == FLT_MAX || (have && !(tm < h.t))) return have;
  const uint32_t om = __reduce_min_sync(FULL, bt == tm ? b_orig : 0xFFFFFFFFu);
  const int f = __ffs((int)__ballot_sync(FULL, bt == tm && b_orig == om)) - 1;
  const int axis = __shfl_sync(FULL, b_axis, f);
  h.m = job_mats + __shfl_sync(FULL, b_mat, f);
  h.t = tm;
  const float s = (axis == 0 ? dx : (axis == 1 ? dy : dz)) > 0.0f ? -1.0f : 1.0f;
  h.nx = axis == 0 ? s : 0.0f;
  h.ny = axis == 1 ? s : 0.0f;
  h.nz = axis == 2 ? s : 0.0f;
  return true;
}

template <int NB, bool TIE, bool WT, bool ALL>
__global__ void __launch_bounds__(kSoloThreads, ALL ? kAllBlocks : kSoloBlocks)
    solo_kernel(const DJob* __restrict__ jobs, uint32_t n_jobs, uint32_t total_rays, const DScene* __restrict__ scenes,
                const DMat* __restrict__ job_mats, const DPanel* __restrict__ panels, float* __restrict__ acc,
                DLaunch* __restrict__ hdr, uint32_t* __restrict__ job_segments, uint32_t max_loop, TailArgs tail) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ SoloShare s_share[ALL ? 1 : kSoloThreads / 32];
  SoloShare& sh = s_share[ALL ? 0 : threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t* err = &hdr->error;
  for (;;) {
    uint32_t rid = 0, ji;
    float px, py, pz, dist, dx, dy, dz, e[NB];
    Pcg rng;
    uint32_t bounce = 0;
    if (tail.rays == nullptr) {
      if (lane == 0) rid = atomicAdd(&hdr->ray_counter, 1u);
      rid = __shfl_sync(FULL, rid, 0);
      if (rid >= total_rays) return;
      ji = find_job(jobs, n_jobs, rid);
      const DJob& J = jobs[ji];
      rng.init(J.seed, rid - J.ray_base);
      unit_sphere(rng, dx, dy, dz);
      px = J.src[0];
      py = J.src[1];
      pz = J.src[2];
      dist = 0.0f;
#pragma unroll
      for (int b = 0; b < NB; b++) e[b] = J.e0[b];
    } else {
      const uint32_t n = hdr->tail;
      if (lane == 0) rid = atomicAdd(&hdr->ended, 1u) - (total_rays - n);
      rid = __shfl_sync(FULL, rid, 0);
      if (rid >= n) return;
      const float4* T = tail.rays + (size_t)kTailWords * rid;
      const float4 a = T[0], d = T[1], c = T[2], e0 = T[3], e1 = T[4];
      px = a.x;
      py = a.y;
      pz = a.z;
      dist = a.w;
      dx = d.x;
      dy = d.y;
      dz = d.z;
      rng.s = __float_as_uint(d.w);
      bounce = __float_as_uint(c.x);
      ji = __float_as_uint(c.y);
      const float ev[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
      for (int b = 0; b < NB; b++) e[b] = ev[b];
    }
    const DJob& J = jobs[ji];
    bool done = false;
    // one segment of the bounce loop (tracer.rs:103-200) a pass; the loop guard counts
    // two a segment, a walk and a shading pass, as a ray in a lane does (trace.cu)
    while (!done) {
      if (bounce >= max_loop / 2u) {
        if (lane == 0) atomicOr(err, 8u);
        return;
      }
      Hit h;
      h.t = FLT_MAX;
      h.m = nullptr;
      bool have;
      if (J.geom == OMG_GEOM_BOX) {
        have = box_hit(J, job_mats, px, py, pz, dx, dy, dz, h);
      } else {
        const DScene& S = scenes[J.scene];
        int prim = -1;
        float t = FLT_MAX;
        if (ALL) have = small_closest<WT>(S, px, py, pz, dx, dy, dz, t, prim, err);
        else have = solo_closest<TIE, WT>(S, sh, px, py, pz, dx, dy, dz, t, prim, err);
        if (have) {
          const float4 p0 = __ldg(S.prims + 3 * (size_t)prim + 0);
          const float4 p1 = __ldg(S.prims + 3 * (size_t)prim + 1);
          const float4 nn = __ldg(S.normals + __float_as_uint(p1.w));
          float nx = nn.x, ny = nn.y, nz = nn.z;
          if (nx * dx + ny * dy + nz * dz > 0.0f) { nx = nx * -1.0f; ny = ny * -1.0f; nz = nz * -1.0f; }
          h.t = t;
          h.nx = nx; h.ny = ny; h.nz = nz;
          h.m = S.mats + __float_as_uint(p0.w);
        }
      }
      if (J.n_panels) have = solo_panels(J, panels, job_mats, px, py, pz, dx, dy, dz, have, h);
      const float t_hit = have ? h.t : FLT_MAX;
      done = shade_segment<NB>(J, acc, h, have, t_hit, px, py, pz, dx, dy, dz, dist, e, rng, lane == 0);
      bounce++;
      if (bounce >= J.max_bounces) done = true;
    }
    if (lane == 0) atomicAdd(job_segments + ji, bounce);
  }
}

}  // namespace

cudaError_t launch_trace_solo(const DJob* jobs, uint32_t n_jobs, uint32_t total_rays, uint32_t max_nb,
                              const DScene* scenes, const DMat* job_mats, const DPanel* panels, float* acc,
                              DLaunch* hdr, uint32_t* job_segments, uint32_t max_loop, int n_sms, bool tie, bool wt,
                              cudaStream_t s, bool small, TailArgs tail) {
  const uint32_t per = kSoloThreads / 32;
  const uint32_t need = ((tail.rays ? tail.cap : total_rays) + per - 1) / per, most = (uint32_t)n_sms * (tie && small ? kAllBlocks : kSoloBlocks);
  const uint32_t blocks = need < most ? need : most;
#define OMG_SOLO(NB, TIE, WT, ALL)                                                                              \
  solo_kernel<NB, TIE, WT, ALL><<<blocks, kSoloThreads, 0, s>>>(jobs, n_jobs, total_rays, scenes, job_mats, panels, \
                                                                acc, hdr, job_segments, max_loop, tail)
#define OMG_SOLO_PICK(NB)                                      \
  if (!tie) OMG_SOLO(NB, false, false, false);                 \
  else if (small && wt) OMG_SOLO(NB, true, true, true);        \
  else if (small) OMG_SOLO(NB, true, false, true);             \
  else if (wt) OMG_SOLO(NB, true, true, false);                \
  else OMG_SOLO(NB, true, false, false)
  if (max_nb <= 3) {
    OMG_SOLO_PICK(3);
  } else {
    OMG_SOLO_PICK(8);
  }
#undef OMG_SOLO_PICK
#undef OMG_SOLO
  return cudaGetLastError();
}

}  // namespace omg
