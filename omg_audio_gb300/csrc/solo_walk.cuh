// One ray's closest hit by a whole warp (the tracer for few rays, the early
// reflections): the 32 lanes take up to 8 pending nodes of the 4-wide tree a
// round, one child box a lane (nodes4c), or 16 of the binary tree (BIN), so a
// round is one load and one slab test deep; the leaves go through the triangle
// test 8 at a time, four lanes each. A lane alone is a chain of some 20 node
// steps of 75 instructions and an L2 trip each on a 50k-primitive scene.
// Nodes, leaves and hits wait in shared memory.
//
// The closest hit is the one the lane walks find. Near-tie rule: it depends
// only on the set of hits (device_common.cuh), so the walk keeps every hit that
// may lie in the final window and takes the lowest key in it at the end.
// First-found rule: the walk goes over the reference's own boxes with its slab
// test, through every leaf that the ray meets, and first_of says which hit the
// reference's ordered walk ends with. Nothing is culled: first_of needs every hit up
// to its bound m, which the last leaf may still move, and a hit's computed distance may
// lie before its own leaf's computed entry, so the nearest hit so far does not say
// which leaves are out (a wider bound would, with such hits left to the lane's walk;
// not built). Where a list is full, one lane walks alone.
#pragma once

#include "device_common.cuh"

namespace omg {

constexpr uint32_t kSoloNodes = 256, kSoloLeaves = 64, kSoloHits = 64;
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

// The near-tie rule's winner among the lanes' candidates (s, tr, t, prim; prim < 0:
// none): the lowest surface, then triangle, then distance. Some lane has one.
__device__ __forceinline__ void tie_winner(uint32_t s, uint32_t tr, float t, int prim, float& t_out, int& prim_out) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t s_min = __reduce_min_sync(FULL, prim >= 0 ? s : 0xFFFFFFFFu);
  bool in = prim >= 0 && s == s_min;
  const uint32_t tr_min = __reduce_min_sync(FULL, in ? tr : 0xFFFFFFFFu);
  in = in && tr == tr_min;
  const uint32_t t_bits = __reduce_min_sync(FULL, in ? __float_as_uint(t) : 0x7f800000u);
  in = in && __float_as_uint(t) == t_bits;
  prim_out = __shfl_sync(FULL, prim, __ffs((int)__ballot_sync(FULL, in)) - 1);
  t_out = __uint_as_float(t_bits);
}

// Meshes of at most kSoloAll primitives (near-tie rule): every lane tests its
// share of them all, which is the set of hits that the walk over the grown boxes
// finds, and the rule depends on that set alone. In a 10 x 7 x 4 m room of few
// triangles the walk's rounds, each a chain of loads, tests and votes, were 6100 of a
// segment's 8200 cycles: 512 rays 340 -> 247 us, 4096 rays 467 -> 455 us (there
// the shading that all lanes repeat is the larger part). 4096 rays in a room of
// 112, 144 and 192 triangles 655, 682, 726 us by the walk; 480 us at 112 with
// this limit, 506, 584, 658 us with 256.
// (A context that lowered the walk budget has its walks counted against it.)
__device__ __forceinline__ bool small_mesh(const DScene& S) {
  return S.n_prims <= kSoloAll && S.walk_budget >= 2u * S.n_nodes + S.n_prims;
}
template <bool WT>
__device__ __noinline__ bool all_closest(const float4* __restrict__ prims, uint32_t n, float ox, float oy, float oz,
                                            float dx, float dy, float dz, float& t_out, int& prim_out) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kEach = (kSoloAll + 31u) / 32u;
  const uint32_t lane = threadIdx.x & 31u;
  float t[kEach], best = FLT_MAX;
  uint32_t s[kEach], tr[kEach];
#pragma unroll
  for (uint32_t r = 0; r < kEach; r++) {
    const uint32_t i = 32u * r + lane;
    t[r] = FLT_MAX;
    if (32u * r < n && i < n) {
      const float4 p0 = __ldg(prims + 3 * (size_t)i), p1 = __ldg(prims + 3 * (size_t)i + 1),
                   p2 = __ldg(prims + 3 * (size_t)i + 2);
      s[r] = __float_as_uint(p2.w);
      tr[r] = __float_as_uint(p1.w);
      float th;
      if (WT ? ray_tri_wt_body(p0, p1, p2, ox, oy, oz, dx, dy, dz, th)
             : ray_tri(p0, p1, p2, ox, oy, oz, dx, dy, dz, th))
        t[r] = th;
    }
    best = fminf(best, t[r]);
  }
  __syncwarp();
  best = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(best)));
  if (best == FLT_MAX) return false;
  const float win = best * (1.0f + kTieRel);
  uint32_t bs = 0, btr = 0;
  float bt = FLT_MAX;
  int prim = -1;
#pragma unroll
  for (uint32_t r = 0; r < kEach; r++)
    if (t[r] < FLT_MAX && t[r] <= win && (prim < 0 || tie_key_less(s[r], tr[r], t[r], bs, btr, bt))) {
      bs = s[r];
      btr = tr[r];
      bt = t[r];
      prim = (int)(32u * r + lane);
    }
  __syncwarp();
  tie_winner(bs, btr, bt, prim, t_out, prim_out);
  return true;
}

// all_closest where it applies, else one lane's walk (a scene that took the slot
// of the one this launch was recorded with).
template <bool WT>
__device__ __forceinline__ bool small_closest(const DScene& S, float ox, float oy, float oz, float dx, float dy,
                                              float dz, float& t_out, int& prim_out, uint32_t* err) {
  constexpr unsigned FULL = 0xffffffffu;
  if (small_mesh(S)) return all_closest<WT>(WT ? S.prims_wt : S.prims, S.n_prims, ox, oy, oz, dx, dy, dz, t_out, prim_out);
  bool have = false;
  float t = 0.0f;
  int prim = 0;
  if ((threadIdx.x & 31u) == 0u) have = lane_closest<true>(S, ox, oy, oz, dx, dy, dz, t, prim, err);
  __syncwarp();
  t_out = __shfl_sync(FULL, t, 0);
  prim_out = __shfl_sync(FULL, prim, 0);
  return __shfl_sync(FULL, (int)have, 0) != 0;
}

// The closest hit of one ray by the whole warp (every argument uniform). BIN:
// over the binary tree (first-found rule only), whose boxes are the reference's
// in every context; nodes4c is exact in first-found contexts alone. A walk that
// runs out of its budget here, where nothing or less is culled, is left to the
// lane's walk.
template <bool TIE, bool WT, bool BIN = false>
__device__ __forceinline__ bool solo_closest(const DScene& S, SoloShare& sh, float ox, float oy, float oz, float dx,
                                             float dy, float dz, float& t_out, int& prim_out, uint32_t* err) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr uint32_t kInf = 0x7f800000u;
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, group = lane >> 2, sub = lane & 3u;
  if (S.n_prims == 0) return false;
  const float4* __restrict__ prims = WT ? S.prims_wt : S.prims;
  if (TIE && small_mesh(S))
    return all_closest<WT>(prims, S.n_prims, ox, oy, oz, dx, dy, dz, t_out, prim_out);
  const float ix = __frcp_rn(dx), iy = __frcp_rn(dy), iz = __frcp_rn(dz);
  // as walk_begin: the slab test by fma (near-tie rule) or minima and maxima
  const float kTiny = 8.673617379884035e-19f;   // 2^-60
  const bool fast = fabsf(ox) <= 7.0f * S.fast_m[0] && fabsf(oy) <= 7.0f * S.fast_m[1] &&
                    fabsf(oz) <= 7.0f * S.fast_m[2] && fabsf(dx) >= kTiny && fabsf(dy) >= kTiny && fabsf(dz) >= kTiny;
  uint32_t nn = 0, nl = 0, nh = 0;
  float best = FLT_MAX;          // the nearest hit so far
  // a list is full; or the tree has no 4-wide form (a launch is chosen by the
  // scenes it was recorded with, and a slot of the scene table may hold another
  // scene by the time it runs)
  bool bail = !BIN && S.root >= 0 && S.nodes4c == nullptr;
  uint32_t budget = S.walk_budget;
  if (S.root >= 0) {
    if (lane == 0) {
      sh.node[0] = BIN ? S.root : S.root4;
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
  while ((nn | nl) != 0u && !bail) {   // (each round takes some of the budget)
    const float cull = TIE ? best * (1.0f + kTieRel) : FLT_MAX;   // (infinite before the first hit)
    if (nl >= 8u || nn == 0u || (nl != 0u && best == FLT_MAX)) {
      // ---- up to 8 leaves, four lanes each
      const uint32_t take = nl < 8u ? nl : 8u, base = nl - take;
      if (budget < take) {
        bail = true;
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
      // ---- up to 8 nodes (BIN: 16), one child a lane
      constexpr uint32_t kTake = BIN ? 16u : 8u;
      const uint32_t take = nn < kTake ? nn : kTake, base = nn - take, g = BIN ? lane >> 1 : group;
      if (budget < take) {
        bail = true;
        break;
      }
      budget -= take;
      const bool act = g < take && sh.node_t[base + (g < take ? g : 0u)] <= cull;
      const int node = act ? sh.node[base + g] : 0;
      nn = base;
      __syncwarp();
      bool h = false;
      float t0 = 0.0f;
      int ref = 0;
      if (act) {
        float4 c0, c1;
        if (BIN) {
          const float4* nd = S.nodes + 4 * (size_t)(uint32_t)node;
          const bool second = (lane & 1u) != 0u;
          const float4 u = __ldg(nd + 1), v = __ldg(nd + (second ? 2 : 0)), n3 = __ldg(nd + 3);
          c0 = second ? make_float4(u.z, u.w, v.x, v.y) : v;
          c1 = second ? make_float4(v.z, v.w, n3.y, 0.0f) : make_float4(u.x, u.y, n3.x, 0.0f);
        } else {
          const float4* nd = S.nodes4c + 8 * (size_t)(uint32_t)node + 2u * sub;
          c0 = __ldg(nd);
          c1 = __ldg(nd + 1);
        }
        ref = __float_as_int(c1.z);
        if (BIN || ref != kEmpty4) {
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
  tie_winner(s, tr, t, prim, t_out, prim_out);
  return true;
}

}  // namespace omg
