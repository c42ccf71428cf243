// Ambient-dome fan on the GPU (crates/omg-scene/src/dome.rs:293-478).
//
// One lane per (listener, fan ray) traces the specular escape
// (trace_escape, dome.rs:330-382: <= max_events mesh hits or pane crossings,
// 80 m horizon); one warp per ray then adds, when the escape is not
// near-full, the straight-through mass-law seep (trace_through,
// dome.rs:390-422, over segment_hits, mesh.rs:546-604). A third kernel bins
// the rays of each listener in fan order (dome.rs:452-458,
// the same f32 sums in the same order), applies the per-listener EMA and
// writes the 9 bins. The fan is deterministic, so the result is too.
#include "cross_walk.cuh"
#include "device_common.cuh"
#include "walk.cuh"

namespace omg {

namespace {

constexpr float PI_F = 3.14159265358979323846f;
constexpr uint32_t kEscBlocks = 7;   // escape blocks a multiprocessor (28 warps, 72 registers)

// dome.rs:56-68
__device__ __forceinline__ bool panel_hit(const DDomePanel& p, float ox, float oy, float oz, float dx, float dy,
                                          float dz, float t_max, float& tout) {
  const float po = p.axis == 0 ? ox : oy, pd = p.axis == 0 ? dx : dy;
  if (fabsf(pd) < 1e-8f) return false;
  const float t = (p.plane - po) / pd;
  if (t < 1e-4f || t >= t_max) return false;
  const float lat = p.axis == 0 ? oy + t * dy : ox + t * dx;
  const float z = oz + t * dz;
  if (lat > p.lat0 && lat < p.lat1 && z > p.z0 && z < p.z1) {
    tout = t;
    return true;
  }
  return false;
}

// The escape of one fan ray as a state machine around its closest-hit walks
// (trace_escape, one event at a time): the ray's position, direction and
// throughput, and how many events it has taken.
template <int NB>
struct EscapeRay {
  float px, py, pz, dx, dy, dz;
  float tp[NB];
  uint32_t ev;
};

// The nearest pane or leaf that a ray crosses before t_max (the first one of
// equal distances; -1: none), one panel a lane (every lane calls this with the
// same ray).
__device__ __forceinline__ int warp_panels(const DDomeLaunch& L, float ox, float oy, float oz, float dx, float dy,
                                           float dz, float t_max, float& tout) {
  constexpr unsigned FULL = 0xffffffffu;
  float bt = t_max;
  int bi = 0x7FFFFFFF;
  for (uint32_t k = threadIdx.x & 31u; k < L.n_panels; k += 32u) {
    float t;
    if (panel_hit(L.panels[k], ox, oy, oz, dx, dy, dz, bt, t)) {
      bt = t;
      bi = (int)k;
    }
  }
  __syncwarp();
  const uint32_t tb = __reduce_min_sync(FULL, bi != 0x7FFFFFFF ? __float_as_uint(bt) : 0x7f800000u);
  const int i = __reduce_min_sync(FULL, bi != 0x7FFFFFFF && __float_as_uint(bt) == tb ? bi : 0x7FFFFFFF);
  tout = __uint_as_float(tb);
  return i == 0x7FFFFFFF ? -1 : i;
}

// One event of trace_escape (dome.rs:336-381) after its closest-hit walk: mesh
// hit (mh, tm, prim) or none, and the nearest panel before it (pan at t_pan, or
// -1). Returns 0 when the ray goes on (the next
// walk starts from its new position), 1 when it escaped, 2 when it ends
// without escaping. The same f32 operations as trace_escape.
template <int NB>
__device__ __forceinline__ int escape_event(const DScene& S, const DDomeLaunch& L, EscapeRay<NB>& r, bool mh, float tm,
                                            int prim, int pan, float t_pan) {
  const uint32_t nb = L.nb;
  if (pan >= 0) {
    const DDomePanel& P = L.panels[pan];
    if (!P.glass) return 2;  // a door leaf blocks
#pragma unroll
    for (int b = 0; b < NB; b++)
      if ((uint32_t)b < nb) r.tp[b] = r.tp[b] * P.t2[b];
    const float adv = t_pan + 1e-3f;
    r.px = r.px + r.dx * adv;
    r.py = r.py + r.dy * adv;
    r.pz = r.pz + r.dz * adv;
    return 0;
  }
  const bool escaped = r.pz > -0.05f || r.dz > 0.05f;
  if (!mh) return escaped ? 1 : 2;
  if (tm > 80.0f) return escaped ? 1 : 2;
  const float4 p0 = __ldg(S.prims + 3 * prim);
  const float4 p1 = __ldg(S.prims + 3 * prim + 1);
  const DMat& M = S.mats[__float_as_uint(p0.w)];
#pragma unroll
  for (int b = 0; b < NB; b++)
    if ((uint32_t)b < nb) r.tp[b] = r.tp[b] * (1.0f - M.absorption[b]);
  if (r.tp[1] < 2e-3f) return 2;
  const float4 nn = __ldg(S.normals + __float_as_uint(p1.w));
  const float nx = nn.x, ny = nn.y, nz = nn.z;
  const float dn = r.dx * nx + r.dy * ny + r.dz * nz;
  float ox = nx, oy = ny, oz = nz;
  if (dn > 0.0f) { ox = nx * -1.0f; oy = ny * -1.0f; oz = nz * -1.0f; }
  const float hx = r.px + r.dx * tm, hy = r.py + r.dy * tm, hz = r.pz + r.dz * tm;
  const float k2 = 2.0f * dn;
  r.dx = r.dx - nx * k2;
  r.dy = r.dy - ny * k2;
  r.dz = r.dz - nz * k2;
  normalize3(r.dx, r.dy, r.dz);
  r.px = hx + ox * 1e-3f;
  r.py = hy + oy * 1e-3f;
  r.pz = hz + oz * 1e-3f;
  return 0;
}

// The specular escape of every (listener, fan ray), one lane each, with the
// persistent tracer's walk: the node phase lane by lane (walk_nodes), then the
// pending leaves tested by the whole warp (coop_leaf_rounds); each event's hit
// is the one any other walk under the context's rule finds, and the events
// follow in the reference's f32 operations (dome.rs:328-382). Lanes from
// rays_per_warp on, and past the last ray, take part in the warp's leaf rounds
// only. A fan of 64 listeners has 32,768 rays, 1024 full warps on 152
// multiprocessors, each waiting on its own loads and on its lanes' divergent
// paths one after another; launch_dome therefore spreads the rays over the
// warps that the chip holds.
// SETTLE: as in trace.cu's trace_kernel.
constexpr uint32_t kEscThreads = 128;
template <int NB, bool TIE, bool WT, bool SETTLE = false>
__global__ void __launch_bounds__(kEscThreads, kEscBlocks) dome_escape_walk_kernel(DDomeLaunch L, uint32_t loop_guard,
                                                                                   uint32_t rays_per_warp) {
  __shared__ uint8_t s_slots[kEscThreads / 32][256];
  const uint32_t total = L.n_eyes * L.n_rays, lane = threadIdx.x & 31u;
  const uint32_t gid = lane < rays_per_warp
                           ? ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * rays_per_warp + lane
                           : 0xFFFFFFFFu;
  const DScene& S = *L.scene;
  uint32_t* err = &L.hdr->error;
  EscapeRay<NB> r{};
  int walk_stack_ref[STACK_DEPTH];
  float walk_stack_t[STACK_DEPTH];
  Walk w;
  w.stack_ref = walk_stack_ref;
  w.stack_t = walk_stack_t;
  w.cur = kDone;
  w.leaf = 0;
  w.prim_best = -1;
  w.t_best = FLT_MAX;
  bool active = gid < total && L.max_events > 0;
  int status = 2;
  uint32_t events = 0;
  if (gid < total) {
    const uint32_t eye = gid / L.n_rays, j = gid % L.n_rays;
    const uint32_t i = (uint32_t)((uint64_t)j * L.n_fan / L.n_rays);  // dome.rs:434
    const float4 f = L.fan[i];
    r.px = L.eyes[3 * eye]; r.py = L.eyes[3 * eye + 1]; r.pz = L.eyes[3 * eye + 2];
    r.dx = f.x; r.dy = f.y; r.dz = f.z;
#pragma unroll
    for (int b = 0; b < NB; b++) r.tp[b] = 1.0f;
    r.ev = 0;
  }
  constexpr unsigned FULL = 0xffffffffu;
  uint32_t iters = 0;
  while (__any_sync(FULL, active)) {
    // the closest hits of every lane's event, then the events together
    bool walking = active;
    if (walking) {
      walk_begin<TIE>(w, S, r.px, r.py, r.pz, r.dx, r.dy, r.dz, false);
      events++;
    }
    while (__any_sync(FULL, walking) && (!TIE || ++iters <= loop_guard)) {
      bool over = false;
      if (walking) {
        int st = 1 << 30;   // the node phase runs until the warp's lanes hold leaves (bounded by the walk budget)
        over = walk_nodes<TIE, SETTLE>(w, S, r.px, r.py, r.pz, st, err);
      }
      coop_leaf_rounds<TIE, WT, SETTLE>(w, walking && !over, WT ? S.prims_wt : S.prims, r.px, r.py, r.pz, r.dx, r.dy,
                                        r.dz, s_slots[threadIdx.x >> 5], kCoopRounds, err);
      if (walking && !over && w.cur == kDone && w.leaf == 0)
        over = !TIE || !walk_restart_fixed(w, S.root, S.walk_budget);
      if (over) walking = false;
    }
    if (iters > loop_guard) {
      atomicOr(err, 8u);
      break;
    }
    if (SETTLE && active) walk_settle(w, S, r.px, r.py, r.pz, r.dx, r.dy, r.dz, err);
    // the panels: each lane its own ray against all of them, or, for few rays,
    // the whole warp on one ray at a time (80 instructions a ray against 25 a panel)
    int pan = -1;
    const float t_mesh = w.prim_best >= 0 ? w.t_best : FLT_MAX;
    float t_pan = t_mesh;
    unsigned rays = __ballot_sync(FULL, active);
    if (3u * (uint32_t)__popc(rays) <= L.n_panels) {
      while (rays) {
        const int o = __ffs((int)rays) - 1;
        rays &= rays - 1u;
        float t;
        const int k = warp_panels(L, __shfl_sync(FULL, r.px, o), __shfl_sync(FULL, r.py, o),
                                  __shfl_sync(FULL, r.pz, o), __shfl_sync(FULL, r.dx, o), __shfl_sync(FULL, r.dy, o),
                                  __shfl_sync(FULL, r.dz, o), __shfl_sync(FULL, t_mesh, o), t);
        if ((int)lane == o) {
          pan = k;
          t_pan = t;
        }
      }
    } else if (active) {
      // a panel whose rectangle misses the segment's box, grown by 1 cm (far more
      // than the crossing's rounding), is not crossed on it: no division (256
      // listeners 806 -> 791 us, 64 391 -> 385)
      float lo[3], hi[3];
      const float p[3] = {r.px, r.py, r.pz}, d[3] = {r.dx, r.dy, r.dz};
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float q = p[a] + d[a] * t_mesh;
        lo[a] = fminf(p[a], q) - 0.01f;
        hi[a] = fmaxf(p[a], q) + 0.01f;
      }
      for (uint32_t k = 0; k < L.n_panels; k++) {
        const DDomePanel& P = L.panels[k];
        const float alo = P.axis == 0 ? lo[0] : lo[1], ahi = P.axis == 0 ? hi[0] : hi[1];
        const float llo = P.axis == 0 ? lo[1] : lo[0], lhi = P.axis == 0 ? hi[1] : hi[0];
        if ((P.plane < alo) | (P.plane > ahi) | (P.lat1 < llo) | (P.lat0 > lhi) | (P.z1 < lo[2]) | (P.z0 > hi[2]))
          continue;
        float t;
        if (panel_hit(L.panels[k], r.px, r.py, r.pz, r.dx, r.dy, r.dz, t_pan, t)) {
          t_pan = t;
          pan = (int)k;
        }
      }
    }
    if (active) {
      const int e = escape_event(S, L, r, walk_have(w), w.t_best, w.prim_best, pan, t_pan);
      r.ev++;
      if (e != 0 || r.ev >= L.max_events) {
        status = e != 0 ? e : 2;
        active = false;
      }
    }
  }
  if (gid < total) {
    float* o = L.ray_tp + (uint64_t)gid * L.nb;
#pragma unroll
    for (int b = 0; b < NB; b++)
      if ((uint32_t)b < L.nb) o[b] = r.tp[b];
    L.ray_escape[gid] = status == 1 ? 1 : 0;
    atomicAdd(&L.events[0], events);
  }
}

// One warp's shared memory for the straight-through segment of one fan ray.
constexpr uint32_t kThroughWarps = 4;        // rays (warps) per block
struct ThroughSmem {
  CrossShare x;
  float st[kMaxCross];                       // crossings sorted
  uint32_t sprim[kMaxCross];
};

// Straight-through seep of one fan ray (trace_through, dome.rs:390-422) by a
// whole warp: the crossings of the 50 m segment (cross_walk.cuh), the
// reference's merge and the transmission product in their order, uniformly
// across the warp.
__device__ void through_warp(const DScene& S, const DDomeLaunch& L, ThroughSmem& W, uint32_t lane, float ex,
                             float ey, float ez, float dx, float dy, float dz, float tp[MAXB]) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t nb = L.nb;
#pragma unroll
  for (int b = 0; b < MAXB; b++) tp[b] = 1.0f;
  const float bx = ex + dx * 50.0f, by = ey + dy * 50.0f, bz = ez + dz * 50.0f;
  if (bz < -0.05f) {
#pragma unroll
    for (int b = 0; b < MAXB; b++) tp[b] = 0.0f;
    return;
  }
  uint32_t n = 0;
  uint32_t fail = 0;   // error bits: 1 walk overflow, 2 too many crossings
  float len = 0.0f;
  if (S.n_prims != 0) {
    float sx = bx - ex, sy = by - ey, sz = bz - ez;
    len = sqrtf(sx * sx + sy * sy + sz * sz);
    if (len >= 1e-6f) {
      const float il = __frcp_rn(len);
      sx = sx * il;
      sy = sy * il;
      sz = sz * il;
      const float ix = __frcp_rn(sx), iy = __frcp_rn(sy), iz = __frcp_rn(sz);
      n = warp_crossings(S, W.x, lane, ex, ey, ez, sx, sy, sz, ix, iy, iz, len, 0xFFFFFFFFu, fail);
    }
  }
  if (fail) {
    if (lane == 0) atomicOr(&L.hdr->error, fail);
#pragma unroll
    for (int b = 0; b < MAXB; b++) tp[b] = 0.0f;
    return;
  }
  for (uint32_t e = lane; e < n; e += 32u) {
    const uint32_t r = cross_rank(W.x, n, e);
    W.st[r] = W.x.t[e];
    W.sprim[r] = W.x.prim[e];
  }
  __syncwarp();
  // same-t merge (lowest surface id wins, the cluster keeps its first t),
  // then the mass-law product in crossing order
  const float tol = 1e-4f / fmaxf(len, 1.0f);
  bool open = false;
  float anchor = 0.0f;
  uint32_t wtri = 0, wmat = 0;
  bool dead = false;
  for (uint32_t q = 0; q <= n && !dead; q++) {
    uint32_t tri = 0, mat = 0;
    float tq = 0.0f;
    const bool last = q == n;
    if (!last) {
      const uint32_t pq = W.sprim[q];
      tq = W.st[q];
      mat = __float_as_uint(__ldg(S.prims + 3 * pq + 0).w);
      tri = __float_as_uint(__ldg(S.prims + 3 * pq + 1).w);
      if (open && fabsf(tq - anchor) < tol) {
        if (S.tri_surface[tri] < S.tri_surface[wtri]) {
          wtri = tri;
          wmat = mat;
        }
        continue;
      }
    }
    if (open) {
      const DMat& M = S.mats[wmat];
#pragma unroll
      for (int b = 0; b < MAXB; b++)
        if ((uint32_t)b < nb) tp[b] = tp[b] * M.t2[b];
      if (tp[0] < 1e-7f) dead = true;
    }
    anchor = tq;
    wtri = tri;
    wmat = mat;
    open = true;
  }
  if (dead) {
#pragma unroll
    for (int b = 0; b < MAXB; b++) tp[b] = 0.0f;
    return;
  }
  // the panels one a lane, then the crossed ones' transmissions in order
  for (uint32_t k0 = 0; k0 < L.n_panels; k0 += 32u) {
    const uint32_t k = k0 + lane;
    float t;
    unsigned crossed =
        __ballot_sync(FULL, k < L.n_panels && panel_hit(L.panels[k], ex, ey, ez, dx, dy, dz, 80.0f, t));
    while (crossed) {
      const DDomePanel& P = L.panels[k0 + (uint32_t)__ffs((int)crossed) - 1u];
      crossed &= crossed - 1u;
#pragma unroll
      for (int b = 0; b < MAXB; b++)
        if ((uint32_t)b < nb) tp[b] = tp[b] * P.t2[b];
    }
  }
}

// dome.rs:432-446 per ray: a near-full escape stands; otherwise the
// straight-through seep, combined with an escape by the per-band max. One
// warp per ray.
__global__ void __launch_bounds__(32 * kThroughWarps) dome_through_kernel(DDomeLaunch L) {
  __shared__ ThroughSmem smem[kThroughWarps];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  const uint64_t gid = (uint64_t)blockIdx.x * kThroughWarps + wib;
  if (gid >= (uint64_t)L.n_eyes * L.n_rays) return;   // warp-uniform
  const uint32_t nb = L.nb;
  float* o = L.ray_tp + gid * nb;
  const bool esc = L.ray_escape[gid] != 0;
  float bp[MAXB];
#pragma unroll
  for (int b = 0; b < MAXB; b++) bp[b] = (uint32_t)b < nb ? o[b] : 0.0f;
  if (esc && bp[0] > 0.5f) return;
  const uint32_t eye = (uint32_t)(gid / L.n_rays), j = (uint32_t)(gid % L.n_rays);
  const uint32_t i = (uint32_t)((uint64_t)j * L.n_fan / L.n_rays);
  const float4 f = L.fan[i];
  const float ex = L.eyes[3 * eye], ey = L.eyes[3 * eye + 1], ez = L.eyes[3 * eye + 2];
  float tp[MAXB];
  through_warp(*L.scene, L, smem[wib], lane, ex, ey, ez, f.x, f.y, f.z, tp);
  if (esc) {
#pragma unroll
    for (int b = 0; b < MAXB; b++) tp[b] = fmaxf(tp[b], bp[b]);
  }
  __syncwarp();
  if (lane == 0) {
    for (uint32_t b = 0; b < nb; b++) o[b] = tp[b];
    atomicAdd(&L.events[1], 1u);
  }
}

// dome.rs:452-477 per listener: bins in fan order, EMA, directions. The
// block stages the listener's rays kDomeChunk at a time: every thread turns
// one ray into its terms (tp / n_rays per band, the direction weighted by
// max(tp[1], 0.2 tp[0]), its bin, or no bin when tp[0] <= 1e-9); then lane
// k < 9 of the first warp adds the terms of bin k's rays in fan order (the
// same f32 sums in the same order as the reference's one loop), finding them
// 32 at a time by ballots.
constexpr uint32_t kDomeChunk = 256;
constexpr uint32_t kDomeBinThreads = 128;
__global__ void __launch_bounds__(kDomeBinThreads) dome_bins_kernel(DDomeLaunch L, float ema_alpha) {
  __shared__ float s_c[kDomeChunk * MAXB];
  __shared__ float s_w[kDomeChunk * 3];
  __shared__ uint32_t s_bin[kDomeChunk];
  const uint32_t eye = blockIdx.x;
  const uint32_t k = threadIdx.x;  // bin 0..8 in the first warp
  const uint32_t nb = L.nb;
  const bool primed = L.primed[eye] != 0u;
  float e[MAXB];
#pragma unroll
  for (int b = 0; b < MAXB; b++) e[b] = 0.0f;
  float sx = 0.0f, sy = 0.0f, sz = 0.0f;
  const float nr = (float)L.n_rays;
  const float* tp_eye = L.ray_tp + (uint64_t)eye * L.n_rays * nb;
  for (uint32_t j0 = 0; j0 < L.n_rays; j0 += kDomeChunk) {
    const uint32_t m = L.n_rays - j0 < kDomeChunk ? L.n_rays - j0 : kDomeChunk;
    for (uint32_t q = threadIdx.x; q < m; q += blockDim.x) {
      const float4 f = L.fan[(uint32_t)((uint64_t)(j0 + q) * L.n_fan / L.n_rays)];
      const float* tp = tp_eye + (uint64_t)(j0 + q) * nb;
      const float t0 = tp[0];
      if (t0 > 1e-9f) {
        for (uint32_t b = 0; b < nb; b++) s_c[q * nb + b] = tp[b] / nr;
        const float w = fmaxf(tp[1], t0 * 0.2f);
        s_w[3 * q] = f.x * w;
        s_w[3 * q + 1] = f.y * w;
        s_w[3 * q + 2] = f.z * w;
        s_bin[q] = (uint32_t)__float_as_int(f.w);
      } else {
        s_bin[q] = 0xFFFFFFFFu;
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      for (uint32_t q0 = 0; q0 < m; q0 += 32) {
        const uint32_t my_bin = q0 + k < m ? s_bin[q0 + k] : 0xFFFFFFFFu;
        uint32_t mine = 0;
        for (uint32_t bin = 0; bin < 9; bin++) {
          const uint32_t bm = __ballot_sync(0xffffffffu, my_bin == bin);
          if (k == bin) mine = bm;
        }
        while (mine) {
          const uint32_t q = q0 + (uint32_t)(__ffs(mine) - 1);
          mine &= mine - 1u;
#pragma unroll
          for (int b = 0; b < MAXB; b++)
            if ((uint32_t)b < nb) e[b] = e[b] + s_c[q * nb + b];
          sx = sx + s_w[3 * q];
          sy = sy + s_w[3 * q + 1];
          sz = sz + s_w[3 * q + 2];
        }
      }
    }
    __syncthreads();
  }
  if (k < 9) {
    const float alpha = primed ? ema_alpha : 1.0f;
    float* ema = L.ema + ((uint64_t)eye * 9 + k) * nb;
    for (uint32_t b = 0; b < nb; b++) {
      L.raw[((uint64_t)eye * 9 + k) * nb + b] = e[b];
      ema[b] = ema[b] + alpha * (e[b] - ema[b]);
      L.out_energy[((uint64_t)eye * 9 + k) * nb + b] = ema[b];
    }
    float dxo, dyo, dzo;
    if (sqrtf(sx * sx + sy * sy + sz * sz) > 1e-6f) {
      dxo = sx; dyo = sy; dzo = sz;
      normalize3(dxo, dyo, dzo);
    } else if (k == 8) {
      dxo = 0.0f; dyo = 0.0f; dzo = 1.0f;
    } else {
      const float az = ((float)k + 0.5f) * TAU_F / 8.0f - PI_F;
      double sn, cs;
      sincos((double)az, &sn, &cs);
      dxo = (float)cs; dyo = (float)sn; dzo = 0.0f;
    }
    float* od = L.out_dir + ((uint64_t)eye * 9 + k) * 3;
    od[0] = dxo;
    od[1] = dyo;
    od[2] = dzo;
  }
  __syncthreads();
  if (k == 0) L.primed[eye] = 1u;
}

// dome.rs:316-324 fan + dome.rs:304-310 bin per direction (in .w)
__global__ void fan_kernel(float4* fan, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float ga = PI_F * (3.0f - sqrtf(5.0f));
  const float z = 1.0f - 2.0f * ((float)i + 0.5f) / (float)n;
  const float r = sqrtf(fmaxf(1.0f - z * z, 0.0f));
  const float phi = ga * (float)i;
  double s, c;
  sincos((double)phi, &s, &c);
  const float x = r * (float)c, y = r * (float)s;
  int bin;
  if (z > 0.87f) {
    bin = 8;
  } else {
    const float az = (float)atan2((double)y, (double)x) + PI_F;
    const float q = az / (TAU_F / 8.0f);
    uint32_t b = q >= 0.0f ? (uint32_t)q : 0u;
    bin = (int)(b < 7u ? b : 7u);
  }
  fan[i] = make_float4(x, y, z, __int_as_float(bin));
}

}  // namespace

cudaError_t build_dome_fan(float4* fan, uint32_t n, cudaStream_t s) {
  fan_kernel<<<(n + 127) / 128, 128, 0, s>>>(fan, n);
  return cudaGetLastError();
}

cudaError_t launch_dome(const DDomeLaunch& L, cudaStream_t s) {
  const uint64_t total = (uint64_t)L.n_eyes * L.n_rays;
  if (total == 0) return cudaSuccess;
  // rays a warp: as few as fill half of the warps that the chip holds. 64
  // listeners (32,768 rays, 16 a warp): 427 us a call, against 439 at 8 and 453
  // at 32; 16 listeners 251 us against 376 with full warps
  const uint64_t warps = (uint64_t)L.n_sms * kEscBlocks * (kEscThreads / 32) / 2u;
  uint32_t rpw = 32;
  while (rpw > 1 && total <= warps * (rpw / 2u)) rpw >>= 1;
  const uint32_t per_block = rpw * (kEscThreads / 32);
  const uint32_t blocks = (uint32_t)((total + per_block - 1) / per_block);
#define OMG_ESCAPE(NB, ...) \
  dome_escape_walk_kernel<NB, __VA_ARGS__><<<blocks, kEscThreads, 0, s>>>(L, kDefaultLoopGuard, rpw)
  if (L.nb <= 3) {
    if (!L.tie && L.capped) OMG_ESCAPE(3, false, false, true);
    else if (!L.tie) OMG_ESCAPE(3, false, false);
    else if (L.wt) OMG_ESCAPE(3, true, true);
    else OMG_ESCAPE(3, true, false);
  } else {
    if (!L.tie && L.capped) OMG_ESCAPE(MAXB, false, false, true);
    else if (!L.tie) OMG_ESCAPE(MAXB, false, false);
    else if (L.wt) OMG_ESCAPE(MAXB, true, true);
    else OMG_ESCAPE(MAXB, true, false);
  }
#undef OMG_ESCAPE
  dome_through_kernel<<<(uint32_t)((total + kThroughWarps - 1) / kThroughWarps), 32 * kThroughWarps, 0, s>>>(L);
  dome_bins_kernel<<<L.n_eyes, kDomeBinThreads, 0, s>>>(L, 0.35f);
  return cudaGetLastError();
}

}  // namespace omg
