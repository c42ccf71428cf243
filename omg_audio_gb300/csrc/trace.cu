// Stochastic energy path tracer kernels for sm_103a.
//
// One persistent kernel traces every ray of every job of a launch: warps pull
// rays from a global queue and refill idle lanes after each segment, so SIMD
// lanes stay busy while rays end at different bounce counts. Each segment is
// one iteration of the reference's bounce loop (tracer.rs:103-200): closest
// hit, receiver test, then absorb / transmit / scatter.
//
// The same kernel also finishes the rays that the wavefront rounds
// (wavefront.cu) leave alive: it then takes ray ids from the tail queue and
// restores each ray's state instead of starting it.
//
// Arithmetic follows the reference's f32 operation order term by term and
// this file is compiled with -fmad=false, so every f32 result rounds exactly
// as the reference's (and the f32 oracle's) does. The only transcendentals,
// cos/sin of the sphere azimuth, come from the f32 sincos of
// device_common.cuh, which the f32 oracle evaluates identically.
#include <algorithm>

#include "shade_common.cuh"
#include "walk.cuh"

namespace omg {

namespace {

// Up to `steps` node visits and leaf tests of a lane on its own; returns true
// when the walk is done.
template <bool TIE>
__device__ __forceinline__ bool walk_steps(Walk& w, const DScene& S, float ox, float oy, float oz, float dx,
                                           float dy, float dz, int steps, bool wide, uint32_t* err) {
  if (TIE && wide && S.nodes4) return walk4_steps(w, S, ox, oy, oz, dx, dy, dz, steps, err);
  if (TIE) return walk_spec(w, S, ox, oy, oz, dx, dy, dz, steps, err);
  return walk_first(w, S, ox, oy, oz, dx, dy, dz, steps, err);
}

// A ray parked between two segments: its state into the per-ray records, for
// the next epoch to restore. (Out of line, as the epoch bookkeeping below: a
// single-launch trace never runs them, and the persistent loop stays small
// enough for the instruction cache.)
template <int NB>
__device__ __noinline__ void park_ray(const WfState& rs, uint32_t rid, float px, float py, float pz, float dist,
                                      float dx, float dy, float dz, uint32_t rng_s, Bands<NB> e, uint32_t bounce) {
  rs.pos[rid] = make_float4(px, py, pz, dist);
  rs.dir[rid] = make_float4(dx, dy, dz, __uint_as_float(rng_s));
  float v[8];
#pragma unroll
  for (int b = 0; b < 8; b++) v[b] = b < NB ? e.v[b] : 0.0f;
  rs.e[rid] = make_float4(v[0], v[1], v[2], v[3]);
  if (NB > 4) rs.e[rs.cap + rid] = make_float4(v[4], v[5], v[6], v[7]);
  rs.bounce[rid] = bounce;
}

// A ray left to the tail launch.
template <int NB>
__device__ __noinline__ void hand_over(float4* rays, uint32_t slot, float px, float py, float pz, float dist, float dx,
                                       float dy, float dz, uint32_t rng_s, Bands<NB> e, uint32_t bounce,
                                       uint32_t job) {
  float4* T = rays + (size_t)kTailWords * slot;
  T[0] = make_float4(px, py, pz, dist);
  T[1] = make_float4(dx, dy, dz, __uint_as_float(rng_s));
  T[2] = make_float4(__uint_as_float(bounce), __uint_as_float(job), 0.0f, 0.0f);
  float v[8];
#pragma unroll
  for (int b = 0; b < 8; b++) v[b] = b < NB ? e.v[b] : 0.0f;
  T[3] = make_float4(v[0], v[1], v[2], v[3]);
  T[4] = make_float4(v[4], v[5], v[6], v[7]);
}

// An epoch's per-iteration bookkeeping, warp-aggregated (every lane calls it):
// count the ended rays (and raise the park signal once at most `keep` remain
// and the queue is drained), append the parked ones to the next epoch's queue.
__device__ __noinline__ void epoch_tally(const EpochArgs& ea, bool ended, bool parked, uint32_t rid, bool may_park,
                                         uint32_t n_rays, uint32_t keep, const uint32_t* fetch) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, lt_mask = (1u << lane) - 1u;
  const unsigned em = __ballot_sync(FULL, ended);
  if (em && lane == (uint32_t)(__ffs(em) - 1)) {
    const uint32_t done_now = atomicAdd(&ea.cur->ended, (uint32_t)__popc(em)) + (uint32_t)__popc(em);
    if (may_park && n_rays - done_now <= keep && *((volatile const uint32_t*)fetch) >= n_rays)
      *((volatile uint32_t*)&ea.cur->park) = 1u;
  }
  const unsigned pm = __ballot_sync(FULL, parked);
  if (pm) {
    uint32_t base = 0;
    if (lane == (uint32_t)(__ffs(pm) - 1)) base = atomicAdd(&ea.next->n, (uint32_t)__popc(pm));
    base = __shfl_sync(FULL, base, __ffs(pm) - 1);
    if (parked) ea.out_q[base + (uint32_t)__popc(pm & lt_mask)] = rid;
  }
}

// The tracer. A lane owns a ray; per loop iteration the warp refills its idle
// lanes from the global ray queue, walks every lane's segment to its closest
// hit, and shades them all together. Walks of a warp differ in length, but the
// shading code is long, and running it for the lanes whose walk is over while
// the others go on walking costs more than the wait (64 pairs on the 40-room
// world: 15 % at groups of 16 lanes), except where walks differ most; and with
// the walk over, none of its state is carried through the shading (64 pairs
// 7.98 -> 8.07 ms, 96 uneven rooms 27.9 -> 27.3 ms, the city 21.6 -> 20.8 ms).
//
// In an epoch chain (ea.cur set) the queue is this epoch's: fresh rays, or
// parked rays whose state is restored from the per-ray records. Once at most
// park_pct % of the epoch's rays remain and its queue is drained, each lane
// parks its ray at the end of its current segment, so that the next epoch
// runs the survivors in full warps. An epoch whose park signal is never
// raised (it ended too few rays while rays were still queued) runs its rays
// to their end, which is only slower.
//
// WIDE (near-tie rule only): walks on the 4-wide tree. A template parameter,
// not a runtime flag, so that each variant carries only its own walk: the
// loop body is then small enough for the instruction cache.
//
// lane_cap: lanes of a warp that take rays (launch_trace: fewer than 32 when
// the launch has fewer rays than the chip has lanes); the other lanes take
// part in the warp's leaf rounds.
//
// Registers: the launch bound (256, 4) caps a thread at 64. Across the loop a
// lane keeps only what the walk reads (the ray, its job, the walk state); the
// segment's hit is computed in the shading pass from the walk's result, and
// the state that only the refill and the shading pass touch (energies,
// distance, stream, segment count, ray id) lives, for up to 4 bands, in shared
// memory, a column per thread. The 3-band near-tie kernel then has 16 bytes of
// spill stores, against 184 with that state in registers.
//
// BOX: every job of a launch without epochs is a shoebox: no walk, every segment
// is one shading pass.
//
// SETTLE: first-found walks that run out of a budget which the caller lowered are
// settled (walk_settle). A variant of its own: the call costs the others 62 bytes of
// spills (64 pairs on the 40-room world, first-found rule, 10.07 -> 10.26 ms).
template <int NB, bool TIE, bool WIDE, bool WT, bool BOX, bool SETTLE = false>
__global__ void __launch_bounds__(256, 4) trace_kernel(const DJob* __restrict__ jobs, uint32_t n_jobs,
                                                       uint32_t total_rays, const DScene* __restrict__ scenes,
                                                       const DMat* __restrict__ job_mats,
                                                       const DPanel* __restrict__ panels,
                                                       const DPanelGroup* __restrict__ groups, float* __restrict__ acc,
                                                    DLaunch* __restrict__ hdr, uint32_t* __restrict__ job_segments,
                                                    uint32_t refill_min, int walk_budget, uint32_t lane_cap,
                                                    EpochArgs ea, TailArgs tail) {
  constexpr bool wide = TIE && WIDE;
  const unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  enum { IDLE = 0, WALK = 1, SHADE = 2 };
  int phase = IDLE;
  bool exhausted = false;
  uint32_t ji = 0;
  float px = 0, py = 0, pz = 0, dx = 0, dy = 0, dz = 0;
  // the ray's state that only the refill and the shading pass touch
  // (energies, distance travelled, stream, segments so far, ray id): for up to
  // 4 bands a column per thread in shared memory, so that it holds no
  // registers across the walk; for 8 bands in registers (there the shared
  // copy's loads and stores in every shading pass cost more than it saves)
  constexpr bool kColdShared = NB <= 4 && !BOX;
  constexpr int kCols = kColdShared ? kMaxWarps * 32 : 1;
  __shared__ float s_e[kColdShared ? NB : 1][kCols];
  __shared__ float s_dist[kCols];
  __shared__ uint32_t s_rng[kCols], s_bounce[kCols], s_rid[kCols];
  const uint32_t me = kColdShared ? threadIdx.x : 0u;
  float r_e[NB];
  float r_dist = 0.0f;
  uint32_t r_rng = 0, r_bounce = 0, r_rid = 0;
  auto cold_save = [&](const float* ev, float dist, uint32_t rng_s, uint32_t bounce) {
#pragma unroll
    for (int b = 0; b < NB; b++) {
      if constexpr (kColdShared) s_e[b][me] = ev[b];
      else r_e[b] = ev[b];
    }
    if constexpr (kColdShared) {
      s_dist[me] = dist;
      s_rng[me] = rng_s;
      s_bounce[me] = bounce;
    } else {
      r_dist = dist;
      r_rng = rng_s;
      r_bounce = bounce;
    }
  };
  auto cold_load = [&](float* ev, float& dist, uint32_t& rng_s, uint32_t& bounce) {
#pragma unroll
    for (int b = 0; b < NB; b++) ev[b] = kColdShared ? s_e[b][me] : r_e[b];
    dist = kColdShared ? s_dist[me] : r_dist;
    rng_s = kColdShared ? s_rng[me] : r_rng;
    bounce = kColdShared ? s_bounce[me] : r_bounce;
  };
  auto cold_set_rid = [&](uint32_t rid) {
    if constexpr (kColdShared) s_rid[me] = rid;
    else r_rid = rid;
  };
  auto cold_rid = [&]() { return kColdShared ? s_rid[me] : r_rid; };
  int walk_stack_ref[STACK_DEPTH];
  float walk_stack_t[STACK_DEPTH];
  uint32_t* err = &hdr->error;
  const WfState& rs = ea.st;
  const bool epoch = !BOX && ea.cur;
  const uint32_t* rq = BOX ? nullptr : ea.in_q;
  const uint32_t n_rays = epoch ? (rq ? ea.cur->n : total_rays) : total_rays;
  uint32_t* fetch = epoch ? &ea.cur->fetch : &hdr->ray_counter;
  const bool may_park = epoch && ea.out_q && n_rays > ea.park_min;
  const uint32_t keep = (uint32_t)(((uint64_t)n_rays * ea.park_pct) / 100u);
  bool parking = false;
  uint32_t iters = 0;   // loop guard (warp-uniform: every lane runs every iteration)
  __shared__ uint8_t s_slots[kMaxWarps][256];   // coop_leaf_rounds' slot lists, one per warp

  // one segment from (p, d): a mesh walk, or (a shoebox) the shading pass
  // alone, which computes the box hit
  auto begin_segment = [&](const DJob& J) { phase = J.geom == OMG_GEOM_BOX ? SHADE : WALK; };

  while (true) {
    if (++iters > ea.max_loop) {
      atomicOr(err, 8u);
      break;
    }
    // ---- refill idle lanes from the ray queue (warp-aggregated)
    const unsigned idle = __ballot_sync(FULL, phase == IDLE && lane < lane_cap);
    if (!exhausted && idle != 0u && (__popc(idle) >= (int)refill_min || __popc(idle) == (int)lane_cap)) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
      base = __shfl_sync(FULL, base, 0);
      // nothing is left for a second fetch; nor where the warps hold every ray of the launch at once
      if (base >= n_rays || (uint32_t)__popc(idle) >= n_rays - base ||
          (uint64_t)gridDim.x * (blockDim.x >> 5) * lane_cap >= n_rays)
        exhausted = true;
      if (phase == IDLE && lane < lane_cap) {
        const uint32_t k = base + (uint32_t)__popc(idle & lt_mask);
        if (k < n_rays) {
          if (rq) {
            const uint32_t rid = rq[k];
            ji = find_job(jobs, n_jobs, rid);
            const float4 P = rs.pos[rid], D = rs.dir[rid];
            px = P.x; py = P.y; pz = P.z;
            dx = D.x; dy = D.y; dz = D.z;
            const float4 e0 = rs.e[rid];
            const float4 e1 = NB > 4 ? rs.e[rs.cap + rid] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float ev[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
            cold_save(ev, P.w, __float_as_uint(D.w), rs.bounce[rid]);
            cold_set_rid(rid);
          } else {
            const uint32_t rid = k;
            ji = find_job(jobs, n_jobs, rid);
            const DJob& J = jobs[ji];
            Pcg rng;
            rng.init(J.seed, rid - J.ray_base);
            unit_sphere(rng, dx, dy, dz);
            px = J.src[0]; py = J.src[1]; pz = J.src[2];
            cold_save(J.e0, 0.0f, rng.s, 0u);
            cold_set_rid(rid);
          }
          begin_segment(jobs[ji]);
        }
      }
    }
    if (__ballot_sync(FULL, phase != IDLE) == 0u) {
      if (exhausted) break;
      continue;
    }
    if (BOX) {
      // No walk, epoch or tail to look at: the lanes' rays on, in registers, until
      // enough lanes wait for new ones (or to their ends, when there are none).
      // A launch that fills the chip is bound by instructions (256 rooms of 8192
      // rays: 6.48 ms with every segment through a loop that also served walks
      // and epochs, 5.99 ms here), a call of few rays by one ray's chain of
      // segments, some 1900 cycles each (1024 rays of 64 segments: 117 us a call
      // through that loop, 106 us here, 96 us with box_hit's quotients side by
      // side and the wall's material loaded ahead of the receiver test).
      float e[NB], dist = 0.0f;
      Pcg rng;
      uint32_t bounce = 0;
      cold_load(e, dist, rng.s, bounce);
      const DJob& J = jobs[ji];
      bool on = phase != IDLE;
      for (;;) {
        if (on) {
          Hit h;
          h.t = FLT_MAX;
          h.m = nullptr;
          bool have = box_hit_body(J, job_mats, px, py, pz, dx, dy, dz, h);
          if (J.n_groups) have = panels_hit(J, panels, groups, job_mats, px, py, pz, dx, dy, dz, have, h);
          const float t_hit = have ? h.t : FLT_MAX;
          const bool done = shade_segment<NB, true>(J, acc, h, have, t_hit, px, py, pz, dx, dy, dz, dist, e, rng);
          bounce++;
          if (done || bounce >= J.max_bounces) {
            atomicAdd(job_segments + ji, bounce);
            on = false;
          }
        }
        const uint32_t live = (uint32_t)__popc(__ballot_sync(FULL, on));
        if (live == 0u || (!exhausted && lane_cap - live >= refill_min)) break;
        if (++iters > ea.max_loop) break;
      }
      cold_save(e, dist, rng.s, bounce);
      phase = on ? SHADE : IDLE;
      continue;
    }
    // the epoch's park signal (sticky; raised only once its queue is drained)
    if (may_park && !parking) parking = *((volatile const uint32_t*)&ea.cur->park) != 0u;

    // ---- the closest-hit walks of every lane's segment, to their end: the
    // node phase lane by lane, then the pending leaves tested by the whole
    // warp together
    int hit_prim = -1;
    float hit_t = FLT_MAX;
    Walk w;
    w.stack_ref = walk_stack_ref;
    w.stack_t = walk_stack_t;
    w.cur = kDone;
    w.leaf = 0;
    bool walking = phase == WALK;
    if (walking) walk_begin<TIE>(w, scenes[jobs[ji].scene], px, py, pz, dx, dy, dz, wide);
    // the loop guard counts the rounds of near-tie walks, and first-found walks once,
    // however many rounds they take: the walk's budget bounds those
    if (!TIE && __any_sync(FULL, walking)) iters++;
    while (__any_sync(FULL, walking)) {
      if (TIE && ++iters > ea.max_loop) break;
      bool over = false;
      if (wide) {
        if (walking)
          over = walk_steps<TIE>(w, scenes[jobs[ji].scene], px, py, pz, dx, dy, dz, walk_budget, wide, err);
      } else {
        const float4* lp = nullptr;
        if (walking) {
          const DScene& S = scenes[jobs[ji].scene];
          lp = WT ? S.prims_wt : S.prims;
          int st = walk_budget;
          over = walk_nodes<TIE, SETTLE>(w, S, px, py, pz, st, err);
        }
        coop_leaf_rounds<TIE, WT, SETTLE>(w, walking && !over, lp, px, py, pz, dx, dy, dz,
                                          s_slots[threadIdx.x >> 5], kCoopRounds, err);
        if (walking && !over && w.cur == kDone && w.leaf == 0) {
          over = true;
          if (TIE) {
            // an ambiguous near-tie window: the walk starts over in fixed mode
            const DScene& S = scenes[jobs[ji].scene];
            over = !walk_restart_fixed(w, S.root, S.walk_budget);
          }
        }
      }
      if (over) walking = false;
    }
    if (iters > ea.max_loop) {
      atomicOr(err, 8u);
      break;
    }
    if (SETTLE && phase == WALK) walk_settle(w, scenes[jobs[ji].scene], px, py, pz, dx, dy, dz, err);
    hit_prim = w.prim_best;
    hit_t = w.t_best;

    // ---- one segment of the bounce loop (tracer.rs:103-200)
    bool ended = false, parked = false;
    if (phase != IDLE) {
      const DJob& J = jobs[ji];
      // the segment's closest hit: the shoebox's, or the walk's (normal of
      // the original triangle, against d)
      Hit h;
      h.t = FLT_MAX;
      h.m = nullptr;
      bool have;
      if (J.geom == OMG_GEOM_BOX) {
        have = box_hit(J, job_mats, px, py, pz, dx, dy, dz, h);
      } else {
        const DScene& S = scenes[J.scene];
        have = hit_prim >= 0;
        if (have) {
          const float4 p0 = __ldg(S.prims + 3 * hit_prim + 0);
          const float4 p1 = __ldg(S.prims + 3 * hit_prim + 1);
          const float4 nn = __ldg(S.normals + __float_as_uint(p1.w));
          float nx = nn.x, ny = nn.y, nz = nn.z;
          if (nx * dx + ny * dy + nz * dz > 0.0f) { nx = nx * -1.0f; ny = ny * -1.0f; nz = nz * -1.0f; }
          h.t = hit_t;
          h.nx = nx; h.ny = ny; h.nz = nz;
          h.m = S.mats + __float_as_uint(p0.w);
        }
      }
      if (J.n_groups) have = panels_hit(J, panels, groups, job_mats, px, py, pz, dx, dy, dz, have, h);
      const float t_hit = have ? h.t : FLT_MAX;
      float e[NB], dist;
      Pcg rng;
      uint32_t bounce;
      cold_load(e, dist, rng.s, bounce);
      bool done = shade_segment<NB>(J, acc, h, have, t_hit, px, py, pz, dx, dy, dz, dist, e, rng);
      bounce++;
      if (!done && bounce >= J.max_bounces) done = true;
      if (done) {
        atomicAdd(job_segments + ji, bounce);
        phase = IDLE;
        ended = true;
      } else if (parking) {
        // save the ray between two segments; the next epoch restores it
        Bands<NB> eb;
#pragma unroll
        for (int b = 0; b < NB; b++) eb.v[b] = e[b];
        park_ray<NB>(rs, cold_rid(), px, py, pz, dist, dx, dy, dz, rng.s, eb, bounce);
        phase = IDLE;
        parked = true;
      } else {
        cold_save(e, dist, rng.s, bounce);
        begin_segment(J);
      }
    }
    if (ea.cur) epoch_tally(ea, ended, parked, cold_rid(), may_park, n_rays, keep, fetch);
    if (tail.rays) {
      // one lane counts and looks, and the warp goes by what it saw: other warps
      // change the counter, and what follows needs all lanes
      const unsigned em = __ballot_sync(FULL, ended);
      uint32_t left = 0;
      if (lane == 0) {
        if (em) atomicAdd(&hdr->ended, (uint32_t)__popc(em));
        left = total_rays - *((volatile const uint32_t*)&hdr->ended);
      }
      left = __shfl_sync(FULL, left, 0);
      if (exhausted && left <= tail.cap) {
        // every ray left in the launch is in some warp: no more than tail.cap are handed over
        const unsigned am = __ballot_sync(FULL, phase != IDLE);
        uint32_t base = 0;
        if (lane == 0 && am) base = atomicAdd(&hdr->tail, (uint32_t)__popc(am));
        base = __shfl_sync(FULL, base, 0);
        if (phase != IDLE) {
          Bands<NB> eb;
          float dist;
          uint32_t rng_s, bounce;
          cold_load(eb.v, dist, rng_s, bounce);
          hand_over<NB>(tail.rays, base + (uint32_t)__popc(am & lt_mask), px, py, pz, dist, dx, dy, dz, rng_s, eb,
                        bounce, ji);
        }
        break;
      }
    }
  }
}

// The tracer as a wavefront inside each warp. A lane walks one ray at a time;
// when its walk ends, the ray id goes to the warp's shading queue and the lane
// takes the next ray to walk from the warp's walk queue (or the global ray
// queue). Once shade_min rays wait in the shading queue (32 by default; or
// nothing is left to walk) the whole warp shades up to 32 of them together,
// from their saved state, and the survivors join the walk queue. Walks thus
// refill lane by lane, and the long shading code runs with full warps (a
// smaller shade_min trades that for shorter waits when few rays are left). A
// warp owns at most 63 rays
// between two fetches from the ray queue (fetching only once its walk queue
// is empty, with at most 31 waiting for shading and 32 walking), so each
// queue holds 64 ids.
//
// Epochs (ea.cur set) work as in trace_kernel: once parking, survivors of a
// shading pass and rays waiting to walk go to the next epoch's queue.
template <int NB, bool TIE>
__global__ void __launch_bounds__(256, 4) trace_wl_kernel(const DJob* __restrict__ jobs, uint32_t n_jobs,
                                                          uint32_t total_rays, const DScene* __restrict__ scenes,
                                                          const DMat* __restrict__ job_mats,
                                                          const DPanel* __restrict__ panels,
                                                          const DPanelGroup* __restrict__ groups,
                                                          float* __restrict__ acc, DLaunch* __restrict__ hdr,
                                                          uint32_t* __restrict__ job_segments, int walk_budget,
                                                          uint32_t shade_min, bool wide, EpochArgs ea) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  constexpr uint32_t kQ = 64;
  __shared__ uint32_t s_shade[8][kQ];
  __shared__ uint32_t s_walk[8][kQ];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t* shade_q = s_shade[threadIdx.x >> 5];
  uint32_t* walk_q = s_walk[threadIdx.x >> 5];
  uint32_t sh_head = 0, sh_cnt = 0, wk_head = 0, wk_cnt = 0;   // warp-uniform
  const WfState& st = ea.st;
  const uint32_t* rq = ea.in_q;
  const uint32_t n_rays = ea.cur ? (rq ? ea.cur->n : total_rays) : total_rays;
  uint32_t* fetch = ea.cur ? &ea.cur->fetch : &hdr->ray_counter;
  const bool may_park = ea.cur && ea.out_q && n_rays > ea.park_min;
  const uint32_t keep = (uint32_t)(((uint64_t)n_rays * ea.park_pct) / 100u);
  bool parking = false, exhausted = false;
  uint32_t* err = &hdr->error;

  // the walking ray of this lane
  uint32_t rid = kNone;
  const DScene* wsc = nullptr;
  float ox = 0, oy = 0, oz = 0, dx = 0, dy = 0, dz = 0;
  int walk_stack_ref[STACK_DEPTH];
  float walk_stack_t[STACK_DEPTH];
  Walk w;
  w.stack_ref = walk_stack_ref;
  w.stack_t = walk_stack_t;

  auto start_walk = [&](uint32_t r) {
    const DJob& J = jobs[find_job(jobs, n_jobs, r)];
    const float4 P = st.pos[r], D = st.dir[r];
    ox = P.x; oy = P.y; oz = P.z;
    dx = D.x; dy = D.y; dz = D.z;
    wsc = scenes + J.scene;
    walk_begin<TIE>(w, *wsc, ox, oy, oz, dx, dy, dz, wide);
    rid = r;
  };
  // ended rays (and the park signal), parked rays to the next epoch's queue
  auto epoch_tally = [&](bool ended, bool parked, uint32_t r) {
    if (!ea.cur) return;
    const unsigned em = __ballot_sync(FULL, ended);
    if (em && lane == (uint32_t)(__ffs(em) - 1)) {
      const uint32_t done_now = atomicAdd(&ea.cur->ended, (uint32_t)__popc(em)) + (uint32_t)__popc(em);
      if (may_park && n_rays - done_now <= keep && *((volatile const uint32_t*)fetch) >= n_rays)
        *((volatile uint32_t*)&ea.cur->park) = 1u;
    }
    const unsigned pm = __ballot_sync(FULL, parked);
    if (pm) {
      uint32_t base = 0;
      if (lane == (uint32_t)(__ffs(pm) - 1)) base = atomicAdd(&ea.next->n, (uint32_t)__popc(pm));
      base = __shfl_sync(FULL, base, __ffs(pm) - 1);
      if (parked) ea.out_q[base + (uint32_t)__popc(pm & lt_mask)] = r;
    }
  };

  uint32_t iters = 0;   // loop guard (warp-uniform)
  while (true) {
    if (++iters > ea.max_loop) {
      atomicOr(err, 8u);
      break;
    }
    // (one lane looks for the warp: another may raise the signal meanwhile, and the passes below need all lanes)
    if (may_park && !parking)
      parking = __shfl_sync(FULL, lane == 0 ? *((volatile const uint32_t*)&ea.cur->park) : 0u, 0) != 0u;
    if (parking && wk_cnt) {
      // rays waiting to walk are between two segments: park them as they are
      const uint32_t m = wk_cnt < 32u ? wk_cnt : 32u;
      const bool pk = lane < m;
      const uint32_t r = pk ? walk_q[(wk_head + lane) % kQ] : kNone;
      wk_head += m;
      wk_cnt -= m;
      epoch_tally(false, pk, r);
      __syncwarp();
      continue;
    }
    unsigned walking = __ballot_sync(FULL, rid != kNone);

    // ---- shading pass: a full warp of rays, or whatever waits once nothing can walk
    if (sh_cnt >= shade_min || (sh_cnt && !walking && !wk_cnt && (exhausted || parking))) {
      const uint32_t m = sh_cnt < 32u ? sh_cnt : 32u;
      bool alive = false, ended = false;
      uint32_t r = kNone;
      if (lane < m) {
        r = shade_q[(sh_head + lane) % kQ];
        alive = shade_saved_ray<NB>(jobs, n_jobs, scenes, job_mats, panels, groups, acc, st, r, job_segments);
        ended = !alive;
      }
      sh_head += m;
      sh_cnt -= m;
      const bool parked = alive && parking;
      alive = alive && !parking;
      const unsigned am = __ballot_sync(FULL, alive);
      if (alive) walk_q[(wk_head + wk_cnt + (uint32_t)__popc(am & lt_mask)) % kQ] = r;
      wk_cnt += (uint32_t)__popc(am);
      epoch_tally(ended, parked, r);
      __syncwarp();
      continue;
    }

    // ---- idle lanes take rays: the walk queue first, then the ray queue
    unsigned idle = ~walking;
    if (idle && wk_cnt) {
      const uint32_t rank = (uint32_t)__popc(idle & lt_mask);
      const uint32_t k = (uint32_t)__popc(idle) < wk_cnt ? (uint32_t)__popc(idle) : wk_cnt;
      if (rid == kNone && rank < k) start_walk(walk_q[(wk_head + rank) % kQ]);
      wk_head += k;
      wk_cnt -= k;
      idle = __ballot_sync(FULL, rid == kNone);
    }
    if (idle && !wk_cnt && !exhausted && !parking) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
      base = __shfl_sync(FULL, base, 0);
      if (base >= n_rays) exhausted = true;
      bool to_shade = false;
      uint32_t r = kNone;
      if (rid == kNone) {
        const uint32_t k = base + (uint32_t)__popc(idle & lt_mask);
        if (k < n_rays) {
          r = rq ? rq[k] : k;
          const DJob& J = jobs[find_job(jobs, n_jobs, r)];
          if (!rq) start_saved_ray<NB>(J, st, r);
          // a shoebox needs no walk: its hit is found when the ray is shaded
          if (J.geom == OMG_GEOM_BOX) to_shade = true;
          else start_walk(r);
        }
      }
      const unsigned bm = __ballot_sync(FULL, to_shade);
      if (to_shade) shade_q[(sh_head + sh_cnt + (uint32_t)__popc(bm & lt_mask)) % kQ] = r;
      sh_cnt += (uint32_t)__popc(bm);
    }
    walking = __ballot_sync(FULL, rid != kNone);
    if (!walking && !sh_cnt && !wk_cnt && (exhausted || parking)) break;

    // ---- walk, at most walk_budget steps this iteration
    bool finished = false;
    if (rid != kNone && walk_steps<TIE>(w, *wsc, ox, oy, oz, dx, dy, dz, walk_budget, wide, err)) {
      st.hit[rid] = make_float2(w.t_best, __int_as_float(w.prim_best));
      finished = true;
    }
    const unsigned fm = __ballot_sync(FULL, finished);
    if (finished) {
      shade_q[(sh_head + sh_cnt + (uint32_t)__popc(fm & lt_mask)) % kQ] = rid;
      rid = kNone;
    }
    sh_cnt += (uint32_t)__popc(fm);
    __syncwarp();
  }
}

// out = (sum + comp) * 2^-64 per float: every job's bins, then every job's dirs.
__global__ void finalize_kernel(const DJob* __restrict__ jobs, uint32_t n_jobs, const float* __restrict__ acc,
                                float* __restrict__ out) {
  const uint32_t j = blockIdx.y;
  if (j >= n_jobs) return;
  const DJob& J = jobs[j];
  const uint32_t nbb = J.n_bins * J.nb, nd = J.n_bins * 3;
  const float* A = acc + J.acc_off;
  float *O = out + J.out_off, *D = out + J.dir_off;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nbb + nd; i += gridDim.x * blockDim.x) {
    float v;
    if (i < nbb) v = A[i] + A[nbb + i];
    else v = A[2 * nbb + (i - nbb)] + A[2 * nbb + nd + (i - nbb)];
    (i < nbb ? O[i] : D[i - nbb]) = v * kAccUnscale;
  }
}

template <bool TIE>
__global__ void raycast_kernel(const DScene* __restrict__ scene, const float* __restrict__ o,
                               const float* __restrict__ d, uint32_t n, float* __restrict__ t_out,
                               uint32_t* __restrict__ tri_out, DLaunch* hdr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const DScene S = *scene;
  float t;
  int prim = 0;
  const float ox = o[3 * i], oy = o[3 * i + 1], oz = o[3 * i + 2];
  const float dx = d[3 * i], dy = d[3 * i + 1], dz = d[3 * i + 2];
  bool have = (TIE && S.nodes4) ? mesh_closest4(S, ox, oy, oz, dx, dy, dz, t, prim, &hdr->error)
                                : mesh_closest<TIE>(S, ox, oy, oz, dx, dy, dz, t, prim, &hdr->error);
  if (have) {
    t_out[i] = t;
    tri_out[i] = __float_as_uint(__ldg(S.prims + 3 * prim + 1).w);
  } else {
    t_out[i] = -1.0f;
    tri_out[i] = 0xFFFFFFFFu;
  }
}

}  // namespace

// Once the ray queue is drained, warps thin out: an iteration with 3 lanes left
// takes 31 us where one with 32 takes 57 (64 pairs on the 40-room world: the last
// 3 % of the rays take 1.2 of 7.5 ms), bound by the chain of one ray's segments.
// A warp on each such ray (solo.cu) is faster from about two rays per resident
// warp down. Calls without a tail, and with one of 28 and 56 rays a
// multiprocessor (ms):
//   rays            16,384  32,768  65,536  262,144  rooms 727,160  city 4,194,304
//   none              3.31    3.73    5.14     7.92          26.72           20.58
//   28 (4256 rays)    3.10    3.40    4.31     7.51          25.25           19.83
//   56 (8512)         3.39    3.55    4.14     7.47          25.07           19.65
// (84 and 112: 7.50 and 7.53 ms at 262,144). Shoeboxes, device-built trees (no
// 4-wide form) and shapes with epochs, rounds or 4-wide walks have none, nor has a
// context with a walk budget of its own, which counts the lanes' visits: a whole warp
// visits other nodes.
uint32_t tail_rays(const LaunchShape& shape, uint32_t total_rays, int n_sms) {
  if (shape.mode != 0 || shape.wide || shape.epochs || shape.wf_iters || !shape.solo_ok || shape.box_only ||
      shape.capped)
    return 0;
  const uint32_t unit = 28u * (uint32_t)n_sms;
  return total_rays < 3u * unit ? 0u : total_rays < 9u * unit ? unit : 2u * unit;
}

cudaError_t launch_trace(const DJob* jobs, uint32_t n_jobs, uint32_t total_rays, uint32_t max_nb,
                         const DScene* scenes, const DMat* job_mats, const DPanel* panels,
                         const DPanelGroup* groups, float* acc, DLaunch* hdr,
                         uint32_t* job_segments, const LaunchShape& shape, int n_sms, bool tie, cudaStream_t s,
                         const EpochArgs* ep, bool wt, float4* tail_buf) {
  if (n_jobs == 0 || total_rays == 0) return cudaSuccess;
  EpochArgs ea{};
  if (ep) ea = *ep;
  // loop iterations of one warp of a persistent kernel before it gives up and
  // flags error 8: by default far above any legitimate count (each iteration
  // advances a walk, a shading pass or the ray queue)
  ea.max_loop = shape.loop_guard ? shape.loop_guard : kDefaultLoopGuard;
  // Few rays on meshes: a warp per ray (solo.cu). Its work per ray is larger, so
  // the lanes win again from about two rays per resident warp: 4096, 8192 and
  // 16,384 rays on the 40-room world 0.72, 1.16 and 1.92 ms against 1.20, 1.51
  // and 1.81 ms (near-tie rule), 0.82, 1.36, 2.18 against 1.51, 1.96, 2.38 ms
  // (first-found rule); on the 12-triangle room 0.46, 0.80, 1.40 against 0.79,
  // 0.89, 1.00 ms. Shoeboxes have no walk to share (a 4096-ray call 0.15
  // against 0.14 ms). A context with a walk budget of its own keeps the lanes (tail_rays).
  if (!ep && !shape.capped && shape.mode == 0 && !shape.wide && shape.solo_ok && !shape.box_only &&
      total_rays <= 2u * 28u * (uint32_t)n_sms)
    return launch_trace_solo(jobs, n_jobs, total_rays, max_nb, scenes, job_mats, panels, acc, hdr, job_segments,
                             ea.max_loop, n_sms, tie, wt, s, shape.small);
  if (shape.mode == 2 && tie && ea.st.pos)
    return launch_trace_coop(jobs, n_jobs, total_rays, max_nb, scenes, job_mats, panels, groups, acc, hdr,
                             job_segments, shape, n_sms, ea, s);
  uint32_t threads = shape.block_threads;
  uint64_t want = (uint64_t)n_sms * shape.blocks_per_sm;
  uint64_t need = ((uint64_t)total_rays + threads - 1) / threads;
  uint32_t blocks = (uint32_t)(want < need ? want : need);
  if (blocks == 0) blocks = 1;
  uint32_t refill = shape.refill_min == 0 ? 1 : (shape.refill_min > 32 ? 32 : shape.refill_min);
  const int steps = shape.walk_steps == 0 ? 1000000 : (int)shape.walk_steps;
  // the warp-local wavefront needs the per-ray records and at most 8 warps a block
  const bool wl = shape.mode == 1 && ea.st.pos && threads <= 256;
  const uint32_t wl_shade = shape.wl_shade_min == 0 ? 32u : (shape.wl_shade_min > 32 ? 32u : shape.wl_shade_min);
  const bool wide = shape.wide != 0;
  // Rays a warp holds at once. A launch with fewer rays than the chip has lanes
  // is bound by one ray's chain of segments: its walk's dependent loads, and
  // the other rays of its warp, whose divergent paths run one after another.
  // So the rays are spread over as many warps as are worth keeping resident
  // (spread_warps a multiprocessor), in blocks of 64 threads so that the
  // multiprocessors get equal shares. Measured (rays: 32 a warp -> this rule):
  // a 64-bounce call on the 40-room world, 4096 rays 3.90 -> 1.37 ms, 65,536
  // rays 4.59 -> 4.28 ms; 200 bounces on the 12-triangle room, 4096 rays
  // 1.37 -> 0.87 ms. At 65,536 rays on the small room 16 a warp is 1.60 ms
  // against 1.53 ms, hence its lower spread_warps.
  uint32_t lane_cap = 32;
  if (!ep) {
    const uint64_t warps = std::min<uint64_t>(want * threads / 32u, (uint64_t)n_sms * shape.spread_warps);
    while (lane_cap > 1 && total_rays <= warps * (lane_cap / 2u)) lane_cap >>= 1;
    if (lane_cap < 32u) {
      const uint32_t spread_threads = threads < 64u ? threads : 64u;
      want = want * threads / spread_threads;
      threads = spread_threads;
      need = ((uint64_t)total_rays * (32u / lane_cap) + threads - 1) / threads;
      blocks = (uint32_t)(want < need ? want : need);
      if (blocks == 0) blocks = 1;
    }
  }
  // Shoebox rays end at different lengths, a lane at a time, and a refill (job
  // lookup, sphere direction) for one lane costs as much as for many: 256 rooms
  // of 8192 rays 6.08, 5.99, 6.04 ms at 4, 6, 8 idle lanes (before the loop kept
  // its rays in registers 7.75, 7.43, 7.08, 6.95, 7.02, 7.41 at 1, 2, 4, 6, 8,
  // 12). Mesh walks are longer: there a lane is refilled at once.
  if (shape.box_only && lane_cap == 32u) refill = std::max(refill, 6u);
  TailArgs tail{nullptr, 0};
  if (!ep && tail_buf) tail = {tail_buf, tail_rays(shape, total_rays, n_sms)};
  if (tail.cap == 0) tail.rays = nullptr;
#define OMG_TRACE_LAUNCH(NB, ...)                                                                            \
  trace_kernel<NB, __VA_ARGS__><<<blocks, threads, 0, s>>>(jobs, n_jobs, total_rays, scenes, job_mats, panels, \
                                                           groups, acc, hdr, job_segments, refill, steps,    \
                                                           lane_cap, ea, tail)
#define OMG_TRACE_PICK(NB)                                                                                    \
  if (wl && tie)                                                                                              \
    trace_wl_kernel<NB, true><<<blocks, threads, 0, s>>>(jobs, n_jobs, total_rays, scenes, job_mats, panels,  \
                                                         groups, acc, hdr, job_segments, steps, wl_shade,     \
                                                         wide, ea);                                           \
  else if (wl)                                                                                                \
    trace_wl_kernel<NB, false><<<blocks, threads, 0, s>>>(jobs, n_jobs, total_rays, scenes, job_mats, panels, \
                                                          groups, acc, hdr, job_segments, steps, wl_shade,    \
                                                          wide, ea);                                          \
  else if (shape.box_only && !ep) OMG_TRACE_LAUNCH(NB, false, false, false, true);                            \
  else if (!tie && shape.capped) OMG_TRACE_LAUNCH(NB, false, false, false, false, true);                      \
  else if (!tie) OMG_TRACE_LAUNCH(NB, false, false, false, false);                                            \
  else if (wide) OMG_TRACE_LAUNCH(NB, true, true, false, false);                                              \
  else if (wt) OMG_TRACE_LAUNCH(NB, true, false, true, false);                                                \
  else OMG_TRACE_LAUNCH(NB, true, false, false, false)
  if (max_nb <= 3) {
    OMG_TRACE_PICK(3);
  } else {
    OMG_TRACE_PICK(8);
  }
#undef OMG_TRACE_PICK
#undef OMG_TRACE_LAUNCH
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !tail.rays) return e;
  return launch_trace_solo(jobs, n_jobs, total_rays, max_nb, scenes, job_mats, panels, acc, hdr, job_segments,
                           ea.max_loop, n_sms, tie, wt, s, shape.small, tail);
}

cudaError_t preload_trace_kernels() {
  cudaFuncAttributes fa;
  cudaError_t e;
  if ((e = cudaFuncGetAttributes(&fa, trace_kernel<3, false, false, false, true>)) != cudaSuccess) return e;
  return cudaFuncGetAttributes(&fa, trace_kernel<8, false, false, false, true>);
}

cudaError_t launch_finalize(const DJob* jobs, uint32_t n_jobs, const float* acc, float* out, uint64_t total_out,
                            cudaStream_t s) {
  if (n_jobs == 0) return cudaSuccess;
  (void)total_out;
  dim3 grid(8, n_jobs);
  finalize_kernel<<<grid, 256, 0, s>>>(jobs, n_jobs, acc, out);
  return cudaGetLastError();
}

cudaError_t launch_raycast(const DScene* scene, const float* o, const float* d, uint32_t n, float* t, uint32_t* tri,
                           DLaunch* hdr, bool tie, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (tie) raycast_kernel<true><<<(n + 127) / 128, 128, 0, s>>>(scene, o, d, n, t, tri, hdr);
  else raycast_kernel<false><<<(n + 127) / 128, 128, 0, s>>>(scene, o, d, n, t, tri, hdr);
  return cudaGetLastError();
}

}  // namespace omg
