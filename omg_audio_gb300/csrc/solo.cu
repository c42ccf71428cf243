// The tracer for launches of few rays: one warp per ray.
//
// What bounds such a launch is one ray's chain of segments, each a chain of
// dependent loads and instructions: a lane walking the binary tree alone takes
// some 25,000 cycles a segment on a 50k-primitive scene (20 node steps of 75
// instructions and an L2 trip each, the leaves, a dozen panel groups), and the
// other lanes of its warp add only divergence. Here the 32 lanes work on one
// ray's segment together:
//   - the walk takes up to 8 pending nodes of the 4-wide tree a round, one
//     child box a lane (nodes4c), so a round is one load and one slab test deep
//     and the tree is half as many levels;
//   - the leaves it meets go through the triangle test 8 at a time, four lanes
//     each;
//   - the panels are tested one a lane;
//   - the shading pass runs uniformly, every lane the same values.
// Nodes, leaves and hits wait in shared memory.
//
// The closest hit is the one the lane walks find. Near-tie rule: it depends
// only on the set of hits (device_common.cuh), so the walk keeps every hit that
// may lie in the final window and takes the lowest key in it at the end.
// First-found rule: the walk goes over the reference's own boxes with its slab
// test, through every leaf that the ray meets (nothing is culled: in the
// reference's order a leaf beyond the nearest hit may come before it), and
// first_of says which hit the reference's ordered walk ends with. Where a list
// is full, one lane walks alone.
#include "shade_common.cuh"

namespace omg {

namespace {

constexpr uint32_t kSoloNodes = 256, kSoloLeaves = 64, kSoloHits = 64;
constexpr uint32_t kSoloThreads = 64;
// Blocks a multiprocessor: 28 warps at 72 registers. (16: 200 bytes of spills,
// 4096 rays on the 40-room world 845 against 811 us; 10 and 8: too few warps
// for 4096 rays, 891 and 1066 us.)
constexpr uint32_t kSoloBlocks = 14;
constexpr float kNearRel = 1e-3f;   // first-found rule: hits kept beyond the nearest
struct SoloShare {
  int node[kSoloNodes];
  float node_t[kSoloNodes];
  int leaf[kSoloLeaves];
  float leaf_t[kSoloLeaves];
  float hit_t[kSoloHits];
  int hit_p[kSoloHits];
  float hit_e[kSoloHits];       // first-found rule: the hit's leaf and its entry distance
  int hit_l[kSoloHits];
};

// The lane walk, for the cases above (called by one lane).
template <bool TIE>
__device__ __noinline__ bool lane_closest(const DScene& S, float ox, float oy, float oz, float dx, float dy, float dz,
                                          float& t, int& prim, uint32_t* err) {
  return mesh_closest<TIE>(S, ox, oy, oz, dx, dy, dz, t, prim, err);
}

// First-found rule: the hit that the reference's ordered walk ends with, from
// the nh nearest hits of all leaves that the ray meets (nearest: `best`; kept up
// to best * (1 + kNearRel)). That walk skips a leaf only when an earlier hit is
// no farther than the leaf's entry. Let m be the least bound such that no leaf
// with a hit within m has its entry beyond m. Hits beyond m then neither win nor
// skip such a leaf, so the walk's end is that of its course over those leaves
// alone: one leaf, mostly; else (coplanar copies of a shared wall) they are
// taken in the walk's order, which the tree above them gives: from the root
// down, the child whose box the ray enters first goes first. Returns false
// where that cannot be told here.
__device__ __forceinline__ bool first_of(const DScene& S, SoloShare& sh, uint32_t nh, float best, bool fast, float ox,
                                         float oy, float oz, float ix, float iy, float iz, float& t_out,
                                         int& prim_out) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  float m = best;
  for (;;) {
    float e = 0.0f;
    for (uint32_t i = lane; i < nh; i += 32u)
      if (sh.hit_t[i] <= m) e = fmaxf(e, sh.hit_e[i]);
    __syncwarp();
    const float em = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(e)));
    if (em <= m) break;
    m = em;
  }
  if (m > best * (1.0f + kNearRel)) return false;
  // those hits, one a lane
  uint32_t n = 0;
  float t = FLT_MAX, e = 0.0f;
  int prim = 0x7FFFFFFF, leaf = 0;
  for (uint32_t i0 = 0; i0 < nh; i0 += 32u) {
    const uint32_t i = i0 + lane;
    const bool in = i < nh && sh.hit_t[i] <= m;
    const unsigned im = __ballot_sync(FULL, in);
    // the k-th of them goes to lane n + k
    const uint32_t k = lane - n;
    const bool mine = lane >= n && k < (uint32_t)__popc(im);
    if (n + (uint32_t)__popc(im) > 32u) return false;
    if (in) sh.leaf[__popc(im & lt)] = (int)i;
    __syncwarp();
    if (mine) {
      const int j = sh.leaf[k];
      t = sh.hit_t[j];
      e = sh.hit_e[j];
      prim = sh.hit_p[j];
      leaf = sh.hit_l[j];
    }
    __syncwarp();
    n += (uint32_t)__popc(im);
  }
  const uint32_t start = ~(uint32_t)leaf >> 3;
  unsigned mask = n >= 32u ? FULL : (1u << n) - 1u;
  int node = S.root;
  uint32_t sp = 0;
  float b_t = FLT_MAX;
  int b_prim = -1;
  for (;;) {
    const int f = __ffs((int)mask) - 1;
    const int l0 = __shfl_sync(FULL, leaf, f);
    if ((__ballot_sync(FULL, leaf == l0) & mask) == mask) {
      // one leaf: tested if its entry is below the best hit; its first nearest primitive
      const bool in = (mask >> lane) & 1u;
      if (__shfl_sync(FULL, e, f) < b_t) {
        const float tm = __uint_as_float(__reduce_min_sync(FULL, in ? __float_as_uint(t) : 0x7f800000u));
        const int pm = __reduce_min_sync(FULL, in && t == tm ? prim : 0x7FFFFFFF);
        if (tm < b_t) {
          b_t = tm;
          b_prim = pm;
        }
      }
      if (sp == 0) break;
      sp--;
      node = sh.node[2 * sp];
      mask = (unsigned)sh.node[2 * sp + 1];
      continue;
    }
    if (node < 0) return false;
    const float4* nd = S.nodes + 4 * (size_t)(uint32_t)node;
    const float4 n3 = __ldg(nd + 3);
    const int c0 = __float_as_int(n3.x), c1 = __float_as_int(n3.y), split = __float_as_int(n3.z);
    if (split < 0) return false;
    const unsigned m0 = __ballot_sync(FULL, start < (uint32_t)split) & mask, m1 = mask & ~m0;
    if (m0 && m1) {
      const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2);
      float ta, tb;
      if (fast) {
        ray_aabb_minmax(n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, ox, oy, oz, ix, iy, iz, FLT_MAX, ta);
        ray_aabb_minmax(n1.z, n1.w, n2.x, n2.y, n2.z, n2.w, ox, oy, oz, ix, iy, iz, FLT_MAX, tb);
      } else {
        ray_aabb(n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, ox, oy, oz, ix, iy, iz, FLT_MAX, ta);
        ray_aabb(n1.z, n1.w, n2.x, n2.y, n2.z, n2.w, ox, oy, oz, ix, iy, iz, FLT_MAX, tb);
      }
      const bool first0 = ta <= tb;
      if (lane == 0) {   // at most one entry a hit: 32
        sh.node[2 * sp] = first0 ? c1 : c0;
        sh.node[2 * sp + 1] = (int)(first0 ? m1 : m0);
      }
      sp++;
      __syncwarp();
      node = first0 ? c0 : c1;
      mask = first0 ? m0 : m1;
    } else {
      node = m0 ? c0 : c1;
    }
  }
  t_out = b_t;
  prim_out = b_prim;
  return true;
}

// The closest hit of one ray by the whole warp (every argument uniform).
template <bool TIE, bool WT>
__device__ __forceinline__ bool solo_closest(const DScene& S, SoloShare& sh, float ox, float oy, float oz, float dx,
                                             float dy, float dz, float& t_out, int& prim_out, uint32_t& iters,
                                             uint32_t max_loop, uint32_t* err) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kInf = 0x7f800000u;
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, group = lane >> 2, sub = lane & 3u;
  if (S.n_prims == 0) return false;
  const float4* __restrict__ prims = WT ? S.prims_wt : S.prims;
  const float ix = __frcp_rn(dx), iy = __frcp_rn(dy), iz = __frcp_rn(dz);
  // as walk_begin: the slab test by fma (near-tie rule) or minima and maxima
  const float kTiny = 8.673617379884035e-19f;   // 2^-60
  const bool fast = fabsf(ox) <= 7.0f * S.fast_m[0] && fabsf(oy) <= 7.0f * S.fast_m[1] &&
                    fabsf(oz) <= 7.0f * S.fast_m[2] && fabsf(dx) >= kTiny && fabsf(dy) >= kTiny && fabsf(dz) >= kTiny;
  uint32_t nn = 0, nl = 0, nh = 0;
  float best = FLT_MAX;          // the nearest hit so far
  bool bail = false;             // a list is full
  uint32_t budget = S.walk_budget;
  if (S.root >= 0) {
    if (lane == 0) {
      sh.node[0] = S.root4;
      sh.node_t[0] = 0.0f;
    }
    nn = 1;
  } else {
    if (lane == 0) {
      sh.leaf[0] = S.root;
      sh.leaf_t[0] = 0.0f;
    }
    nl = 1;
  }
  __syncwarp();
  while ((nn | nl) != 0u && !bail) {
    if (++iters > max_loop) break;
    const float cull = TIE ? best * (1.0f + kTieRel) : FLT_MAX;   // (infinite before the first hit)
    if (nl >= 8u || nn == 0u || (nl != 0u && best == FLT_MAX)) {
      // ---- up to 8 leaves, four lanes each
      const uint32_t take = nl < 8u ? nl : 8u, base = nl - take;
      if (budget < take) {
        if (lane == 0) atomicOr(err, 4u);
        break;
      }
      budget -= take;
      const bool act = group < take;
      const int lf = act ? sh.leaf[base + group] : 0;
      const float t0 = act ? sh.leaf_t[base + group] : 0.0f;
      nl = base;
      const uint32_t code = ~(uint32_t)lf, start = code >> 3, cnt = act && t0 <= cull ? (code & 7u) + 1u : 0u;
      for (uint32_t k = sub; __any_sync(FULL, k < cnt); k += 4u) {
        bool hit = false;
        float t = 0.0f;
        if (k < cnt) {
          const float4* P = prims + 3 * (size_t)(start + k);
          const float4 p0 = __ldg(P), p1 = __ldg(P + 1), p2 = __ldg(P + 2);
          hit = WT ? ray_tri_wt_body(p0, p1, p2, ox, oy, oz, dx, dy, dz, t)
                   : ray_tri(p0, p1, p2, ox, oy, oz, dx, dy, dz, t);
        }
        if (!__any_sync(FULL, hit)) continue;
        const float tm = __uint_as_float(__reduce_min_sync(FULL, hit ? __float_as_uint(t) : kInf));
        best = fminf(best, tm);
        const bool keep = hit && t <= best * (1.0f + (TIE ? kTieRel : kNearRel));
        const unsigned km = __ballot_sync(FULL, keep);
        if (nh + (uint32_t)__popc(km) > kSoloHits) {
          bail = true;
          break;
        }
        if (keep) {
          const uint32_t at = nh + (uint32_t)__popc(km & lt);
          sh.hit_t[at] = t;
          sh.hit_p[at] = (int)(start + k);
          if (!TIE) {
            sh.hit_e[at] = t0;
            sh.hit_l[at] = lf;
          }
        }
        nh += (uint32_t)__popc(km);
      }
      __syncwarp();
    } else {
      // ---- up to 8 nodes, one child a lane
      const uint32_t take = nn < 8u ? nn : 8u, base = nn - take;
      if (budget < take) {
        if (lane == 0) atomicOr(err, 4u);
        break;
      }
      budget -= take;
      const bool act = group < take && sh.node_t[base + (group < take ? group : 0u)] <= cull;
      const int node = act ? sh.node[base + group] : 0;
      nn = base;
      __syncwarp();
      bool h = false;
      float t0 = 0.0f;
      int ref = 0;
      if (act) {
        const float4* nd = S.nodes4c + 8 * (size_t)(uint32_t)node + 2u * sub;
        const float4 c0 = __ldg(nd), c1 = __ldg(nd + 1);
        ref = __float_as_int(c1.z);
        if (ref != kEmpty4) {
          if (!fast)
            h = ray_aabb(c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, ox, oy, oz, ix, iy, iz, cull, t0);
          else if (TIE)
            h = ray_aabb_fma(c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, ox * ix, oy * iy, oz * iz, ix, iy, iz, cull, t0);
          else
            h = ray_aabb_minmax(c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, ox, oy, oz, ix, iy, iz, cull, t0);
        }
      }
      const unsigned lm = __ballot_sync(FULL, h && ref < 0), nm = __ballot_sync(FULL, h && ref >= 0);
      if (nn + (uint32_t)__popc(nm) > kSoloNodes) {
        bail = true;
        break;
      }
      if (h) {
        const uint32_t at = ref < 0 ? nl + (uint32_t)__popc(lm & lt) : nn + (uint32_t)__popc(nm & lt);
        (ref < 0 ? sh.leaf : sh.node)[at] = ref;
        (ref < 0 ? sh.leaf_t : sh.node_t)[at] = t0;
      }
      nl += (uint32_t)__popc(lm);   // fewer than 8 before: 40 at most
      nn += (uint32_t)__popc(nm);
      __syncwarp();
    }
  }
  if (!TIE && !bail && nh != 0u) {
    if (first_of(S, sh, nh, best, fast, ox, oy, oz, ix, iy, iz, t_out, prim_out)) return true;
    bail = true;
  }
  if (bail) {
    bool have = false;
    float t = 0.0f;
    int prim = 0;
    if (lane == 0) have = lane_closest<TIE>(S, ox, oy, oz, dx, dy, dz, t, prim, err);
    __syncwarp();
    t_out = __shfl_sync(FULL, t, 0);
    prim_out = __shfl_sync(FULL, prim, 0);
    return __shfl_sync(FULL, (int)have, 0) != 0;
  }
  if (nh == 0) return false;
  // the lowest (surface, triangle, t) in the window
  const float win = best * (1.0f + kTieRel);
  uint32_t s = 0xFFFFFFFFu, tr = 0xFFFFFFFFu;
  float t = FLT_MAX;
  int prim = -1;
  for (uint32_t i = lane; i < nh; i += 32u) {
    const float ti = sh.hit_t[i];
    if (ti > win) continue;
    const int pi = sh.hit_p[i];
    const uint32_t si = __float_as_uint(__ldg(&prims[3 * (size_t)pi + 2].w)),
                   tri = __float_as_uint(__ldg(&prims[3 * (size_t)pi + 1].w));
    if (prim < 0 || tie_key_less(si, tri, ti, s, tr, t)) {
      s = si;
      tr = tri;
      t = ti;
      prim = pi;
    }
  }
  __syncwarp();
  const uint32_t s_min = __reduce_min_sync(FULL, prim >= 0 ? s : 0xFFFFFFFFu);
  bool in = prim >= 0 && s == s_min;
  const uint32_t tr_min = __reduce_min_sync(FULL, in ? tr : 0xFFFFFFFFu);
  in = in && tr == tr_min;
  const uint32_t t_bits = __reduce_min_sync(FULL, in ? __float_as_uint(t) : kInf);
  in = in && __float_as_uint(t) == t_bits;
  prim_out = __shfl_sync(FULL, prim, __ffs((int)__ballot_sync(FULL, in)) - 1);
  t_out = __uint_as_float(t_bits);
  return true;
}

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

template <int NB, bool TIE, bool WT>
__global__ void __launch_bounds__(kSoloThreads, kSoloBlocks)
    solo_kernel(const DJob* __restrict__ jobs, uint32_t n_jobs, uint32_t total_rays, const DScene* __restrict__ scenes,
                const DMat* __restrict__ job_mats, const DPanel* __restrict__ panels, float* __restrict__ acc,
                DLaunch* __restrict__ hdr, uint32_t* __restrict__ job_segments, uint32_t max_loop) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ SoloShare s_share[kSoloThreads / 32];
  SoloShare& sh = s_share[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t* err = &hdr->error;
  uint32_t iters = 0;   // loop guard
  while (iters <= max_loop) {
    uint32_t rid = 0;
    if (lane == 0) rid = atomicAdd(&hdr->ray_counter, 1u);
    rid = __shfl_sync(FULL, rid, 0);
    if (rid >= total_rays) return;
    const uint32_t ji = find_job(jobs, n_jobs, rid);
    const DJob& J = jobs[ji];
    Pcg rng;
    rng.init(J.seed, rid - J.ray_base);
    float dx, dy, dz;
    unit_sphere(rng, dx, dy, dz);
    float px = J.src[0], py = J.src[1], pz = J.src[2], dist = 0.0f;
    float e[NB];
#pragma unroll
    for (int b = 0; b < NB; b++) e[b] = J.e0[b];
    uint32_t bounce = 0;
    bool done = false;
    // one segment of the bounce loop (tracer.rs:103-200) a pass
    while (!done && ++iters <= max_loop) {
      Hit h;
      h.t = FLT_MAX;
      h.m = nullptr;
      bool have;
      if (J.geom == OMG_GEOM_BOX) {
        have = box_hit_body(J, job_mats, px, py, pz, dx, dy, dz, h);
      } else {
        const DScene& S = scenes[J.scene];
        int prim = -1;
        float t = FLT_MAX;
        have = solo_closest<TIE, WT>(S, sh, px, py, pz, dx, dy, dz, t, prim, iters, max_loop, err);
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
    if (lane == 0 && done) atomicAdd(job_segments + ji, bounce);
  }
  if (lane == 0) atomicOr(err, 8u);
}

}  // namespace

cudaError_t launch_trace_solo(const DJob* jobs, uint32_t n_jobs, uint32_t total_rays, uint32_t max_nb,
                              const DScene* scenes, const DMat* job_mats, const DPanel* panels, float* acc,
                              DLaunch* hdr, uint32_t* job_segments, uint32_t max_loop, int n_sms, bool tie, bool wt,
                              cudaStream_t s) {
  const uint32_t per = kSoloThreads / 32;
  const uint32_t need = (total_rays + per - 1) / per, most = (uint32_t)n_sms * kSoloBlocks;
  const uint32_t blocks = need < most ? need : most;
#define OMG_SOLO(NB, TIE, WT)                                                                                      \
  solo_kernel<NB, TIE, WT><<<blocks, kSoloThreads, 0, s>>>(jobs, n_jobs, total_rays, scenes, job_mats, panels, acc, \
                                                           hdr, job_segments, max_loop)
  if (max_nb <= 3) {
    if (!tie) OMG_SOLO(3, false, false);
    else if (wt) OMG_SOLO(3, true, true);
    else OMG_SOLO(3, true, false);
  } else {
    if (!tie) OMG_SOLO(8, false, false);
    else if (wt) OMG_SOLO(8, true, true);
    else OMG_SOLO(8, true, false);
  }
#undef OMG_SOLO
  return cudaGetLastError();
}

}  // namespace omg
