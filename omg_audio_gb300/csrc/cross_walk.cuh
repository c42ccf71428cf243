// The crossings of a segment by a whole warp (segment_hits, mesh.rs:546-604;
// the dome's straight-through segments, the early reflections' legs).
//
// An any-hit walk visits every node that the segment meets. Every lane takes one
// pending node a round (children whose box the segment meets are pushed
// warp-aggregated), so the walk runs 32 nodes wide instead of one. Leaves wait in
// a list of their own and are tested eight at a time, four lanes each: a lane that
// met a leaf among the nodes tested its primitives alone, in nearly every round.
// Near the end of the list the walk takes as few nodes as there is room for, at
// last one, the reference's own order, which needs no more than the tree's depth.
//
// The reference sorts the crossings by t with a stable sort over its
// depth-first visiting order (child b before child a) and then merges
// clusters within 1e-4 / max(len, 1) keeping the lowest surface id (the
// first one on equal ids). Each ref therefore carries its depth-first
// position: bit 63 - d set for the a child at depth d (d < 58) above a
// 6-bit depth, so that ordering crossings by (t, key, primitive) reproduces
// the reference's order.
#pragma once

#include "device_common.cuh"

namespace omg {

constexpr uint32_t kMaxCross = 64;           // crossings kept per segment
constexpr uint32_t kCrossStack = 384;        // pending nodes of one warp's walk
constexpr uint32_t kCrossLeaves = 72;        // pending leaves (fewer than 8, and a round's 64 children)

// One warp's shared memory.
struct CrossShare {
  unsigned long long key[kCrossStack];       // the ref's depth-first position
  unsigned long long lkey[kCrossLeaves];
  unsigned long long ckey[kMaxCross];
  int ref[kCrossStack];
  int lref[kCrossLeaves];
  float t[kMaxCross];                        // crossings as found
  uint32_t prim[kMaxCross];
  uint32_t n;
};

// The crossings of a + t d, t in (0, len) (d a unit vector, i its reciprocals;
// every argument uniform), as found: their number. fail: error bits 1 (list of
// nodes full), 2 (more than kMaxCross crossings), 4 (more than `budget` visits).
__device__ __forceinline__ uint32_t warp_crossings(const DScene& S, CrossShare& W, uint32_t lane, float ax, float ay,
                                                   float az, float dx, float dy, float dz, float ix, float iy,
                                                   float iz, float len, uint32_t budget, uint32_t& fail) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t lt = (1u << lane) - 1u;
  constexpr float kTiny = 8.673617379884035e-19f;   // 2^-60: no product of the slab test is a NaN
  const bool fast = fabsf(dx) >= kTiny && fabsf(dy) >= kTiny && fabsf(dz) >= kTiny;
  uint32_t sp = S.root >= 0 ? 1u : 0u, nl = 1u - sp;
  __syncwarp();   // the last segment's crossings have been read
  if (lane == 0) {
    (sp ? W.ref : W.lref)[0] = S.root;
    (sp ? W.key : W.lkey)[0] = 0ull;
    W.n = 0u;
  }
  __syncwarp();
  while ((sp | nl) != 0u) {
    if (nl >= 8u || sp == 0u) {
      // ---- up to 8 leaves, four lanes each
      const uint32_t take = nl < 8u ? nl : 8u, g = lane >> 2;
      if (budget < take) {
        fail |= 4u;
        break;
      }
      budget -= take;
      nl -= take;
      const bool act = g < take;
      const uint32_t code = act ? ~(uint32_t)W.lref[nl + g] : 0u;
      const uint32_t start = code >> 3, cnt = act ? (code & 7u) + 1u : 0u;
      for (uint32_t k = lane & 3u; __any_sync(FULL, k < cnt); k += 4u) {
        if (k >= cnt) continue;
        const uint32_t i = start + k;
        const float4 p0 = __ldg(S.prims + 3 * i + 0);
        const float4 p1 = __ldg(S.prims + 3 * i + 1);
        const float4 p2 = __ldg(S.prims + 3 * i + 2);
        float t;
        if (ray_tri(p0, p1, p2, ax, ay, az, dx, dy, dz, t)) {
          const float tt = t / len;
          if (tt > 1e-4f && tt < 1.0f - 1e-4f) {
            const uint32_t q = atomicAdd(&W.n, 1u);
            if (q < kMaxCross) {
              W.t[q] = tt;
              W.prim[q] = i;
              W.ckey[q] = W.lkey[nl + g];
            }
          }
        }
      }
      __syncwarp();
      continue;
    }
    // ---- up to 32 nodes, one a lane
    const uint32_t room = kCrossStack - STACK_DEPTH > sp ? kCrossStack - STACK_DEPTH - sp : 1u;
    const uint32_t take = min(min(sp, 32u), room);
    if (budget < take) {
      fail |= 4u;
      break;
    }
    budget -= take;
    const uint32_t base = sp - take;
    const bool act = lane < take;
    int cur = 0;
    unsigned long long key = 0ull;
    if (act) {
      cur = W.ref[base + lane];
      key = W.key[base + lane];
    }
    __syncwarp();
    sp = base;
    bool h0 = false, h1 = false;
    int c0 = 0, c1 = 0;
    if (act) {
      const float4 n0 = __ldg(S.nodes + 4 * cur + 0);
      const float4 n1 = __ldg(S.nodes + 4 * cur + 1);
      const float4 n2 = __ldg(S.nodes + 4 * cur + 2);
      const float4 n3 = __ldg(S.nodes + 4 * cur + 3);
      float ta, tb;
      if (fast) {
        h0 = ray_aabb_minmax(n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, ax, ay, az, ix, iy, iz, len, ta);
        h1 = ray_aabb_minmax(n1.z, n1.w, n2.x, n2.y, n2.z, n2.w, ax, ay, az, ix, iy, iz, len, tb);
      } else {
        h0 = ray_aabb(n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, ax, ay, az, ix, iy, iz, len, ta);
        h1 = ray_aabb(n1.z, n1.w, n2.x, n2.y, n2.z, n2.w, ax, ay, az, ix, iy, iz, len, tb);
      }
      c0 = __float_as_int(n3.x);
      c1 = __float_as_int(n3.y);
    }
    const unsigned m0 = __ballot_sync(FULL, h0 && c0 >= 0), m1 = __ballot_sync(FULL, h1 && c1 >= 0);
    const unsigned l0 = __ballot_sync(FULL, h0 && c0 < 0), l1 = __ballot_sync(FULL, h1 && c1 < 0);
    const uint32_t tot = (uint32_t)(__popc(m0) + __popc(m1));
    if (sp + tot > kCrossStack) {
      fail |= 1u;
      break;
    }
    const uint32_t d = (uint32_t)(key & 63ull);
    const unsigned long long child = (key & ~63ull) | (unsigned long long)(d < 63u ? d + 1u : 63u);
    const unsigned long long abit = d < 58u ? (1ull << (63u - d)) : 0ull;
    if (h0) {
      const uint32_t at = c0 < 0 ? nl + (uint32_t)__popc(l0 & lt) : sp + (uint32_t)__popc(m0 & lt);
      (c0 < 0 ? W.lref : W.ref)[at] = c0;
      (c0 < 0 ? W.lkey : W.key)[at] = child | abit;
    }
    if (h1) {
      const uint32_t at = c1 < 0 ? nl + (uint32_t)(__popc(l0) + __popc(l1 & lt))
                                 : sp + (uint32_t)(__popc(m0) + __popc(m1 & lt));
      (c1 < 0 ? W.lref : W.ref)[at] = c1;
      (c1 < 0 ? W.lkey : W.key)[at] = child;
    }
    sp += tot;
    nl += (uint32_t)(__popc(l0) + __popc(l1));
    __syncwarp();
  }
  __syncwarp();
  const uint32_t n = W.n;
  if (n > kMaxCross) fail |= 2u;
  return n;
}

// Crossing e's place in the reference's order (every key is distinct).
__device__ __forceinline__ uint32_t cross_rank(const CrossShare& W, uint32_t n, uint32_t e) {
  const float te = W.t[e];
  const unsigned long long ke = W.ckey[e];
  const uint32_t pe = W.prim[e];
  uint32_t r = 0;
  for (uint32_t q = 0; q < n; q++) {
    const float tq = W.t[q];
    const unsigned long long kq = W.ckey[q];
    if (tq < te || (tq == te && (kq < ke || (kq == ke && W.prim[q] < pe)))) r++;
  }
  return r;
}

}  // namespace omg
