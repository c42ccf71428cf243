// World early reflections on the GPU (crates/omg-core/src/pt_mesh.rs).
//
// Discovery (mesh_chains, pt_mesh.rs:382-457): every fan ray bounces
// specularly off the mesh and the furniture boxes up to 3 times; every
// surface chain it passes is a candidate. A global hash table keeps, per
// chain, the lowest candidate index (ray-major, bounce-minor: the order in
// which the reference's sequential loop meets them), and one block compacts
// the first occurrences in that order, which is the reference's output order.
//
// Solve (mesh_record, pt_mesh.rs:186-337): every (source, chain) pair mirrors
// the source across the chain's planes, validates each bounce by a closest-hit
// query (the reference's first-found order over the binary tree) and pays the
// transmission of every surface and blocker each leg crosses (segment_hits,
// mesh.rs:546-604: crossings in depth-first order, stably sorted by t, equal-t
// clusters merged to the lowest surface id).
//
// What bounds both is one ray's or pair's chain of dependent node loads: a call
// has some 768 rays, and few of its pairs (340 of 25,600 on the 40-room world)
// are paths. Discovery gives each ray a warp of its own until the resident warps
// have two, and lanes of its own warp beyond (one thread per ray, 24 full warps:
// 213 us for 768 rays on that world; spread 52 us). The path's planes, sides and
// directions follow from geometry alone, so a thread per pair settles those
// first (8 us for the 25,600), and a warp walks each pair that is left (closest
// hits by solo_walk.cuh, crossings by cross_walk.cuh): 176 us, where a thread per
// pair that did it all took 461 us, the same spread over more warps 440 us, and
// warps over all pairs that pass the first closest hit 401 us (17,169 of them: a
// wall in front ends a path only if it lets nothing through).
//
// f32 arithmetic in the reference's operation order (built with -fmad=false,
// IEEE division and square root); cos/sin of the fan azimuth and exp of the
// air attenuation are evaluated in double and rounded once.
#include <algorithm>
#include <cfloat>

#include "cross_walk.cuh"
#include "device_common.cuh"
#include "solo_walk.cuh"

namespace omg {

namespace {

constexpr uint16_t kNoSurf = 0xFFFFu;

__device__ __forceinline__ float dot3(const float a[3], float x, float y, float z) {
  return a[0] * x + a[1] * y + a[2] * z;
}

__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf(x * x + y * y + z * z); }

__device__ __forceinline__ bool dead3(const float v[3], float lim) { return v[0] < lim && v[1] < lim && v[2] < lim; }

// One warp's shared memory: a closest hit's lists, or a segment's walk and its
// merged crossings.
struct WarpShare {
  union {
    SoloShare solo;
    CrossShare x;
  };
  float t[kMaxCross];
  uint32_t sid[kMaxCross], mat[kMaxCross];
};

// Closest hit in the reference's first-found order: (t, original triangle,
// material) or false. Alone, or (WARP) by the whole warp with the same arguments
// in every lane, over the binary tree: its boxes are the reference's in every
// context.
template <bool WARP>
__device__ __forceinline__ bool raycast_ref(const DEarly& E, SoloShare* sh, float ox, float oy, float oz, float dx,
                                            float dy, float dz, float& t, uint32_t& tri, uint32_t& mat) {
  int prim = 0;
  bool have;
  if (WARP) {
    have = solo_closest<false, false, true>(E.S, *sh, ox, oy, oz, dx, dy, dz, t, prim, E.err);
    __syncwarp();
  } else {
    have = mesh_closest<false>(E.S, ox, oy, oz, dx, dy, dz, t, prim, E.err);
  }
  if (!have) return false;
  mat = __float_as_uint(__ldg(E.S.prims + 3 * prim + 0).w);
  tri = __float_as_uint(__ldg(E.S.prims + 3 * prim + 1).w);
  return true;
}

// ------------------------------------------------------------- discovery
constexpr uint32_t kDiscThreads = 64;
constexpr uint32_t kDiscBlocks = 14;         // blocks, 28 warps a multiprocessor

struct DiscArgs {
  DEarly E;
  float lx, ly, lz;
  uint32_t n_rays, rot, rays_per_warp;
  uint32_t use_boxes;
  float ga;                           // golden angle, f32 (pt_mesh.rs:392)
  const float* jitter;                // the rotation's xorshift draws, one per ray
  unsigned long long* cand_key;
  omg_chain* cand_chain;
  uint32_t* cand_slot;
  unsigned long long* tkey;
  uint32_t* tidx;
  uint32_t tcap;
};

__device__ __forceinline__ uint32_t key_hash(unsigned long long k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  return (uint32_t)k;
}

// Candidate j: the first k + 1 surfaces of a ray's chain.
__device__ __forceinline__ void place_candidate(const DiscArgs& A, uint32_t j, int k, const uint16_t* chain) {
  unsigned long long key = 1ull;
  for (int q = 0; q <= k; q++) key = key * 65536ull + (unsigned long long)chain[q] + 1ull;
  A.cand_key[j] = key;
  omg_chain c;
  for (int q = 0; q < OMG_CHAIN_MAX_ORDER; q++) c.surf[q] = chain[q];
  c.order = (uint16_t)(k + 1);
  A.cand_chain[j] = c;
  // first occurrence per key: the lowest candidate index (its complement, so that
  // the table is cleared to zeros throughout)
  uint32_t h = key_hash(key) & (A.tcap - 1u);
  bool placed = false;
  for (uint32_t probe = 0; probe < A.tcap; probe++) {
    const unsigned long long prev = atomicCAS(A.tkey + h, 0ull, key);
    if (prev == 0ull || prev == key) {
      atomicMax(A.tidx + h, ~j);
      A.cand_slot[j] = h;
      placed = true;
      break;
    }
    h = (h + 1u) & (A.tcap - 1u);
  }
  if (!placed) {
    atomicOr(A.E.err, 8u);
    A.cand_key[j] = 0ull;
  }
}

// WARP: a warp per ray, every lane with the same values; else rays_per_warp
// lanes of a warp a ray each.
template <bool WARP>
__global__ void __launch_bounds__(kDiscThreads, kDiscBlocks) early_discover_kernel(DiscArgs A) {
  __shared__ SoloShare s_solo[WARP ? kDiscThreads / 32 : 1];
  const uint32_t lane = threadIdx.x & 31u, warp = (blockIdx.x * kDiscThreads + threadIdx.x) >> 5;
  SoloShare* sh = &s_solo[WARP ? threadIdx.x >> 5 : 0];
  const uint32_t i = WARP ? warp : warp * A.rays_per_warp + lane;
  if ((!WARP && lane >= A.rays_per_warp) || i >= A.n_rays) return;
  const bool lead = !WARP || lane == 0u;
  const DEarly& E = A.E;
  if (lead)
    for (int k = 0; k < OMG_CHAIN_MAX_ORDER; k++) A.cand_key[3 * i + k] = 0ull;
  const float z = 1.0f - 2.0f * ((float)i + 0.5f) / (float)A.n_rays;
  const float r = sqrtf(fmaxf(1.0f - z * z, 0.0f));
  const float phi = A.ga * (float)i + (float)A.rot * 0.61803398875f * 6.28318530717958647692f + A.jitter[i] * 0.02f;
  double sd, cd;
  sincos((double)phi, &sd, &cd);
  float dx = r * (float)cd, dy = r * (float)sd, dz = z;
  float px = A.lx, py = A.ly, pz = A.lz;
  uint16_t chain[OMG_CHAIN_MAX_ORDER] = {kNoSurf, kNoSurf, kNoSurf};
  for (int k = 0; k < OMG_CHAIN_MAX_ORDER; k++) {
    float t = FLT_MAX, nx = 0.0f, ny = 0.0f, nz = 1.0f;
    bool has = false;
    uint32_t sid = 0;
    {
      float mt;
      uint32_t tri, mat;
      if (raycast_ref<WARP>(E, sh, px, py, pz, dx, dy, dz, mt, tri, mat)) {
        t = mt;
        has = true;
        sid = E.S.tri_surface[tri];
        const float4 nn = __ldg(E.S.normals + tri);
        nx = nn.x;
        ny = nn.y;
        nz = nn.z;
      }
    }
    if (A.use_boxes) {
      const float p[3] = {px, py, pz}, d[3] = {dx, dy, dz};
      for (uint32_t bi = 0; bi < E.n_boxes; bi++) {
        const float4 bl = __ldg(E.boxes + 2 * bi), bh = __ldg(E.boxes + 2 * bi + 1);
        const float mn[3] = {bl.x, bl.y, bl.z}, mx[3] = {bh.x, bh.y, bh.z};
        float t0 = 1e-4f, t1 = t;
        int axis = 3;
        for (int a = 0; a < 3; a++) {
          const float da = d[a];
          if (fabsf(da) < 1e-9f) {
            if (p[a] < mn[a] || p[a] > mx[a]) {
              t0 = FLT_MAX;
              break;
            }
          } else {
            float ta = (mn[a] - p[a]) / da, tb = (mx[a] - p[a]) / da;
            if (ta > tb) {
              const float q = ta;
              ta = tb;
              tb = q;
            }
            if (ta > t0) {
              t0 = ta;
              axis = a;
            }
            t1 = fminf(t1, tb);
            if (t0 > t1) {
              t0 = FLT_MAX;
              break;
            }
          }
        }
        if (t0 < t && axis < 3) {
          t = t0;
          const int face = axis * 2 + (d[axis] > 0.0f ? 0 : 1);
          has = true;
          sid = (E.base_overlay + bi * 6u + (uint32_t)face) & 0xFFFFu;
          nx = ny = nz = 0.0f;
          const float s = d[axis] > 0.0f ? -1.0f : 1.0f;
          if (axis == 0) nx = s;
          else if (axis == 1) ny = s;
          else nz = s;
        }
      }
    }
    if (!has) break;
    if (t <= 1e-4f || t > 200.0f) break;
    px = px + dx * t;
    py = py + dy * t;
    pz = pz + dz * t;
    chain[k] = (uint16_t)sid;
    if (lead) place_candidate(A, 3u * i + (uint32_t)k, k, chain);
    // specular bounce off the hit normal, faced against the ray
    const float dn0 = nx * dx + ny * dy + nz * dz;
    if (dn0 > 0.0f) {
      nx = nx * -1.0f;
      ny = ny * -1.0f;
      nz = nz * -1.0f;
    }
    const float s2 = 2.0f * (dx * nx + dy * ny + dz * nz);
    dx = dx - nx * s2;
    dy = dy - ny * s2;
    dz = dz - nz * s2;
    px = px + nx * 1e-4f;
    py = py + ny * 1e-4f;
    pz = pz + nz * 1e-4f;
  }
}

// One block: the first occurrences, compacted in candidate order.
constexpr uint32_t kCompactThreads = 1024;
__global__ void __launch_bounds__(kCompactThreads)
    early_compact_kernel(const unsigned long long* __restrict__ cand_key, const omg_chain* __restrict__ cand_chain,
                         const uint32_t* __restrict__ cand_slot, const uint32_t* __restrict__ tidx, uint32_t n_cand,
                         omg_chain* out, uint32_t cap, uint32_t* n_out) {
  __shared__ uint32_t warp_tot[kCompactThreads / 32];
  __shared__ uint32_t base;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) base = 0;
  __syncthreads();
  for (uint32_t chunk = 0; chunk < n_cand; chunk += kCompactThreads) {
    const uint32_t j = chunk + tid;
    const bool keep = j < n_cand && cand_key[j] != 0ull && tidx[cand_slot[j]] == ~j;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_tot[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (warp == 0) {
      const uint32_t v = warp_tot[lane];
      uint32_t incl = v;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += u;
      }
      warp_tot[lane] = incl - v;   // exclusive prefix of the warps
    }
    __syncthreads();
    const uint32_t pos = base + warp_tot[warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (keep && pos < cap) out[pos] = cand_chain[j];
    __syncthreads();
    if (tid == kCompactThreads - 1) base = pos + (keep ? 1u : 0u);
    __syncthreads();
  }
  if (tid == 0) *n_out = base;
}

// ----------------------------------------------------------------- solve
// mesh.rs:546-604 by a warp: every crossing of a->b strictly between its ends,
// in the reference's order, merged, into W.t / W.sid / W.mat. Their number.
__device__ uint32_t segment_hits(const DEarly& E, float ax, float ay, float az, float bx, float by, float bz,
                                 WarpShare& W) {
  const DScene& S = E.S;
  const uint32_t lane = threadIdx.x & 31u;
  if (S.n_prims == 0) return 0;
  float dx = bx - ax, dy = by - ay, dz = bz - az;
  const float len = len3(dx, dy, dz);
  if (len < 1e-6f) return 0;
  const float il = __frcp_rn(len);
  dx = dx * il;
  dy = dy * il;
  dz = dz * il;
  const float ix = __frcp_rn(dx), iy = __frcp_rn(dy), iz = __frcp_rn(dz);
  float tr;
  if (!ray_aabb(E.root_lo[0], E.root_lo[1], E.root_lo[2], E.root_hi[0], E.root_hi[1], E.root_hi[2], ax, ay, az, ix,
                iy, iz, len, tr))
    return 0;
  uint32_t fail = 0;
  const uint32_t n = warp_crossings(S, W.x, lane, ax, ay, az, dx, dy, dz, ix, iy, iz, len, S.walk_budget, fail);
  if (fail) {
    if (lane == 0) atomicOr(E.err, fail);
    return 0;
  }
  for (uint32_t e = lane; e < n; e += 32u) {
    const uint32_t r = cross_rank(W.x, n, e), prim = W.x.prim[e];
    W.t[r] = W.x.t[e];
    W.sid[r] = S.tri_surface[__float_as_uint(__ldg(S.prims + 3 * prim + 1).w)];
    W.mat[r] = __float_as_uint(__ldg(S.prims + 3 * prim + 0).w);
  }
  __syncwarp();
  // same-t clusters: the lowest surface id wins, the cluster keeps its first t
  // (a crossing is written at or before its own place, by one lane)
  const float tol = 1e-4f / fmaxf(len, 1.0f);
  uint32_t w = 0;
  if (lane == 0) {
    for (uint32_t i = 0; i < n; i++) {
      const float t = W.t[i];
      const uint32_t sid = W.sid[i], mat = W.mat[i];
      if (w > 0 && fabsf(t - W.t[w - 1]) < tol) {
        if (sid < W.sid[w - 1]) {
          W.sid[w - 1] = sid;
          W.mat[w - 1] = mat;
        }
      } else {
        W.t[w] = t;
        W.sid[w] = sid;
        W.mat[w] = mat;
        w++;
      }
    }
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, w, 0);
}

// pt.rs:43-70
__device__ __forceinline__ bool aabb_clip(const omg_aabb& x, float ax, float ay, float az, float bx, float by,
                                          float bz) {
  const float a[3] = {ax, ay, az}, d[3] = {bx - ax, by - ay, bz - az};
  float t0 = 0.0f, t1 = 1.0f;
  for (int k = 0; k < 3; k++) {
    if (fabsf(d[k]) < 1e-9f) {
      if (a[k] < x.mn[k] || a[k] > x.mx[k]) return false;
    } else {
      float ta = (x.mn[k] - a[k]) / d[k], tb = (x.mx[k] - a[k]) / d[k];
      if (ta > tb) {
        const float q = ta;
        ta = tb;
        tb = q;
      }
      t0 = fmaxf(t0, ta);
      t1 = fminf(t1, tb);
      if (t0 > t1) return false;
    }
  }
  return t1 > 1e-4f && t0 < 1.0f - 1e-4f;
}

// pt_mesh.rs:146-182, by a warp: what the crossings and the blockers let
// through, a lane each for the tests and the loads, in their order for the product.
__device__ bool leg_transmission(const DEarly& E, float ax, float ay, float az, float bx, float by, float bz,
                                 bool has_skip, uint32_t skip_sid, float t_expect, const omg_aabb* extras,
                                 uint32_t n_extras, WarpShare& W, float tr[3]) {
  constexpr unsigned FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t n = segment_hits(E, ax, ay, az, bx, by, bz, W);
  const float seg_len = fmaxf(len3(bx - ax, by - ay, bz - az), 1e-6f);
  for (uint32_t i0 = 0; i0 < n; i0 += 32u) {
    const uint32_t i = i0 + lane;
    float4 m = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    bool on = false;
    if (i < n) {
      on = !(has_skip && W.sid[i] == skip_sid && fabsf(W.t[i] - t_expect) * seg_len < 0.05f);
      m = __ldg(E.mtrans + W.mat[i]);
    }
    unsigned left = __ballot_sync(FULL, on);
    while (left) {
      const int f = __ffs((int)left) - 1;
      left &= left - 1u;
      tr[0] = tr[0] * __shfl_sync(FULL, m.x, f);
      tr[1] = tr[1] * __shfl_sync(FULL, m.y, f);
      tr[2] = tr[2] * __shfl_sync(FULL, m.z, f);
      if (dead3(tr, 1e-6f)) return false;
    }
  }
  for (uint32_t k0 = 0; k0 < n_extras; k0 += 32u) {
    unsigned left = __ballot_sync(FULL, k0 + lane < n_extras && aabb_clip(extras[k0 + lane], ax, ay, az, bx, by, bz));
    while (left) {
      const omg_aabb& x = extras[k0 + (uint32_t)__ffs((int)left) - 1u];
      left &= left - 1u;
      for (int b = 0; b < 3; b++) tr[b] = tr[b] * x.transmission[b];
      if (dead3(tr, 1e-6f)) return false;
    }
  }
  return true;
}

// The start of mesh_record: the source mirrored across the chain's planes, the
// listener's distance and direction to that image. False: no path.
__device__ __forceinline__ bool image_of(const DEarly& E, const omg_chain& ch, float sx, float sy, float sz, float lx,
                                         float ly, float lz, float& dist, float& dirx, float& diry, float& dirz) {
  float ix = sx, iy = sy, iz = sz;
  for (int i = (int)ch.order - 1; i >= 0; i--) {
    if (ch.surf[i] >= E.n_surf) return false;
    const DSurf& s = E.surf[ch.surf[i]];
    const float k = 2.0f * (dot3(s.n, ix, iy, iz) - s.d);
    ix = ix - s.n[0] * k;
    iy = iy - s.n[1] * k;
    iz = iz - s.n[2] * k;
  }
  const float tx = ix - lx, ty = iy - ly, tz = iz - lz;
  dist = len3(tx, ty, tz);
  if (dist < 1e-4f) return false;
  const float idist = __frcp_rn(dist);
  dirx = tx * idist;
  diry = ty * idist;
  dirz = tz * idist;
  return true;
}

// Where the leg (p, d) meets the bounce's plane, and whether a furniture
// face's rectangle holds the point. False: no path.
__device__ __forceinline__ bool plane_hit(const DSurf& s, float px, float py, float pz, float dx, float dy, float dz,
                                          float& t, float& hx, float& hy, float& hz) {
  const float denom = dot3(s.n, dx, dy, dz);
  if (fabsf(denom) < 1e-9f) return false;
  t = (s.d - dot3(s.n, px, py, pz)) / denom;
  if (t <= 1e-4f) return false;
  hx = px + dx * t;
  hy = py + dy * t;
  hz = pz + dz * t;
  if (s.rect) {
    const float eps = 1e-3f;
    const float h[3] = {hx, hy, hz};
    for (int a = 0; a < 3; a++)
      if (h[a] < s.fmin[a] - eps || h[a] > s.fmax[a] + eps) return false;
  }
  return true;
}

// On from the bounce at h: the specular direction, off the surface by 1e-4.
__device__ __forceinline__ void bounce_off(const DSurf& s, float hx, float hy, float hz, float& px, float& py,
                                           float& pz, float& dx, float& dy, float& dz) {
  const float nd = dot3(s.n, dx, dy, dz);
  const float off = nd < 0.0f ? 1e-4f : -1e-4f;
  px = hx + s.n[0] * off;
  py = hy + s.n[1] * off;
  pz = hz + s.n[2] * off;
  const float k2 = 2.0f * nd;
  dx = dx - s.n[0] * k2;
  dy = dy - s.n[1] * k2;
  dz = dz - s.n[2] * k2;
}

// After the last bounce: the source on this side of its plane, and ahead.
__device__ __forceinline__ bool same_side(const DEarly& E, const omg_chain& ch, float px, float py, float pz, float sx,
                                          float sy, float sz) {
  if (ch.order == 0) return true;
  const DSurf& s = E.surf[ch.surf[ch.order - 1]];
  return !((dot3(s.n, px, py, pz) - s.d) * (dot3(s.n, sx, sy, sz) - s.d) < 0.0f);
}
__device__ __forceinline__ bool ahead(const omg_chain& ch, float px, float py, float pz, float dx, float dy, float dz,
                                      float sx, float sy, float sz) {
  if (ch.order == 0) return true;
  const float qx = sx - px, qy = sy - py, qz = sz - pz;
  const float leg = len3(qx, qy, qz);
  if (!(leg > 1e-4f)) return true;
  const float il = __frcp_rn(leg);
  return !((qx * il) * dx + (qy * il) * dy + (qz * il) * dz < 0.995f);
}

// What geometry alone says of a pair: false where mesh_record finds no path
// whatever its walks find.
__device__ __forceinline__ bool path_stands(const DEarly& E, const omg_chain& ch, float sx, float sy, float sz,
                                            float lx, float ly, float lz) {
  float dist, dx, dy, dz;
  if (!image_of(E, ch, sx, sy, sz, lx, ly, lz, dist, dx, dy, dz)) return false;
  float px = lx, py = ly, pz = lz;
  for (int i = 0; i < (int)ch.order; i++) {
    const DSurf& s = E.surf[ch.surf[i]];
    float t, hx, hy, hz;
    if (!plane_hit(s, px, py, pz, dx, dy, dz, t, hx, hy, hz)) return false;
    bounce_off(s, hx, hy, hz, px, py, pz, dx, dy, dz);
  }
  return same_side(E, ch, px, py, pz, sx, sy, sz) && ahead(ch, px, py, pz, dx, dy, dz, sx, sy, sz);
}

// The leg's closest hit against the bounce at t: the bounce stands, ends the
// path, or lies behind something that lets sound through (the leg's crossings
// then have to show the surface).
enum Cast { kCastDead, kCastStands, kCastBehind };
template <bool WARP>
__device__ __forceinline__ Cast cast_of(const DEarly& E, SoloShare* sh, const DSurf& s, uint32_t sid, float t, float px, float py,
                                        float pz, float dx, float dy, float dz) {
  float rt;
  uint32_t rtri, rmat;
  const bool hit =
      raycast_ref<WARP>(E, sh, px + dx * 1e-4f, py + dy * 1e-4f, pz + dz * 1e-4f, dx, dy, dz, rt, rtri, rmat);
  if (s.rect) {
    if (!hit || !(rt < t - 1e-3f)) return kCastStands;
    const float4 m = __ldg(E.mtrans + rmat);
    const float mt[3] = {m.x, m.y, m.z};
    return dead3(mt, 1e-6f) ? kCastDead : kCastStands;
  }
  if (!hit) return kCastDead;
  if (E.S.tri_surface[rtri] == sid && fabsf(rt - t) < 2e-2f) return kCastStands;
  if (!(rt < t - 1e-3f)) return kCastDead;
  const float4 m = __ldg(E.mtrans + rmat);
  const float mt[3] = {m.x, m.y, m.z};
  return dead3(mt, 1e-4f) ? kCastDead : kCastBehind;
}

// The same by a warp with one result: all lanes together, or the first alone.
template <bool WARP>
__device__ __forceinline__ Cast warp_cast(const DEarly& E, WarpShare& W, const DSurf& s, uint32_t sid, float t,
                                          float px, float py, float pz, float dx, float dy, float dz) {
  if (WARP) return cast_of<true>(E, &W.solo, s, sid, t, px, py, pz, dx, dy, dz);
  int c = 0;
  if ((threadIdx.x & 31u) == 0u) c = cast_of<false>(E, nullptr, s, sid, t, px, py, pz, dx, dy, dz);
  __syncwarp();
  return (Cast)__shfl_sync(0xffffffffu, c, 0);
}

// pt_mesh.rs:186-337, by a warp (every lane with the same arguments and values)
template <bool WARP>
__device__ bool mesh_record(const DEarly& E, const omg_chain& ch, uint16_t source, float sx, float sy, float sz,
                            float lx, float ly, float lz, const omg_aabb* extras, uint32_t n_extras, WarpShare& W,
                            omg_mesh_record& out) {
  const int order = ch.order;
  float dist, dirx, diry, dirz;
  if (!image_of(E, ch, sx, sy, sz, lx, ly, lz, dist, dirx, diry, dirz)) return false;
  float gm[3] = {1.0f, 1.0f, 1.0f};
  float px = lx, py = ly, pz = lz, dx = dirx, dy = diry, dz = dirz;
  for (int i = 0; i < order; i++) {
    const uint32_t sid = ch.surf[i];
    if (sid >= E.n_surf) return false;
    const DSurf& s = E.surf[sid];
    float t, hx, hy, hz;
    if (!plane_hit(s, px, py, pz, dx, dy, dz, t, hx, hy, hz)) return false;
    const Cast cast = warp_cast<WARP>(E, W, s, sid, t, px, py, pz, dx, dy, dz);
    if (cast == kCastDead) return false;
    if (cast == kCastBehind) {
      const uint32_t n = segment_hits(E, px, py, pz, hx + dx * 0.05f, hy + dy * 0.05f, hz + dz * 0.05f, W);
      bool found = false;
      for (uint32_t q = 0; q < n; q++)
        if (W.sid[q] == sid && fabsf(W.t[q] * (t + 0.05f) - t) < 0.1f) found = true;
      if (!found) return false;
    }
    if (!leg_transmission(E, px, py, pz, hx, hy, hz, true, sid, 1.0f, extras, n_extras, W, gm)) return false;
    for (int b = 0; b < 3; b++) gm[b] = gm[b] * s.refl[b];
    bounce_off(s, hx, hy, hz, px, py, pz, dx, dy, dz);
  }
  if (!same_side(E, ch, px, py, pz, sx, sy, sz)) return false;
  if (!leg_transmission(E, px, py, pz, sx, sy, sz, false, 0u, 0.0f, extras, n_extras, W, gm)) return false;
  if (!ahead(ch, px, py, pz, dx, dy, dz, sx, sy, sz)) return false;
  const float dtot = fmaxf(dist, 0.3f);
  const float kAir[3] = {1.0e-4f, 5.0e-4f, 3.0e-3f};  // AIR_ABSORPTION_PER_M, material.rs:76
  float gains[3];
  for (int b = 0; b < 3; b++) {
    const float air = (float)exp((double)(-kAir[b] * dtot));
    gains[b] = air / dtot * gm[b];
  }
  if (dead3(gains, 2e-5f)) return false;
  out.source = source;
  for (int q = 0; q < OMG_CHAIN_MAX_ORDER; q++) out.chain[q] = q < order ? ch.surf[q] : kNoSurf;
  out.order = (uint32_t)order;
  out.delay_s = dist / 343.0f;
  out.dir[0] = dirx;
  out.dir[1] = diry;
  out.dir[2] = dirz;
  for (int b = 0; b < 3; b++) out.gains[b] = gains[b];
  uint32_t h = 0x811C9DC5u ^ (uint32_t)source;
  for (int q = 0; q < order; q++) h = (h ^ (uint32_t)ch.surf[q]) * 16777619u;
  out.key = (h ^ 0xA5u) * 16777619u;
  out.valid = 1u;
  return true;
}

constexpr uint32_t kSolveThreads = 64;
constexpr uint32_t kSolveBlocks = 12;        // 24 warps a multiprocessor (14, 9: 512 sources 1539, 1644 against 1533 us)
constexpr uint32_t kSiftThreads = 128;

struct SolveArgs {
  DEarly E;
  const uint16_t* ids;
  const float* pos;
  uint32_t n_src;
  const omg_chain* chains;
  uint32_t n_chains;
  float lx, ly, lz;
  const omg_aabb* extras;
  uint32_t n_extras;
  uint64_t first;        // this launch's pairs: first .. first + n - 1
  uint32_t n;
  uint32_t* live;        // [0] pairs that need walks, then their numbers less `first`
  omg_mesh_record* out;
};

__device__ __forceinline__ void no_record(omg_mesh_record& r, uint16_t source, const omg_chain& ch) {
  r.source = source;
  for (int q = 0; q < OMG_CHAIN_MAX_ORDER; q++) r.chain[q] = ch.surf[q];
  r.order = ch.order;
  r.delay_s = 0.0f;
  r.dir[0] = r.dir[1] = r.dir[2] = 0.0f;
  r.gains[0] = r.gains[1] = r.gains[2] = 0.0f;
  r.key = 0u;
  r.valid = 0u;
}

// A thread per pair: what the pair's geometry decides without a walk. Pairs that
// end there get their empty record; the others are listed. (All of them where the
// context has a walk budget of its own, which the walks of every pair count against.)
__global__ void __launch_bounds__(kSiftThreads) early_sift_kernel(SolveArgs A) {
  const uint32_t i = blockIdx.x * kSiftThreads + threadIdx.x, lane = threadIdx.x & 31u;
  bool live = false;
  if (i < A.n) {
    const uint64_t k = A.first + i;
    const uint32_t s = (uint32_t)(k / A.n_chains), c = (uint32_t)(k % A.n_chains);
    const omg_chain ch = A.chains[c];
    live = A.E.capped || path_stands(A.E, ch, A.pos[3 * s], A.pos[3 * s + 1], A.pos[3 * s + 2], A.lx, A.ly, A.lz);
    if (!live) no_record(A.out[k], A.ids[s], ch);
  }
  __syncwarp();
  const unsigned m = __ballot_sync(0xffffffffu, live);
  uint32_t base = 0;
  if (lane == 0 && m) base = atomicAdd(A.live, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (live) A.live[1u + base + (uint32_t)__popc(m & ((1u << lane) - 1u))] = i;
}

// A warp per listed pair.
template <bool WARP>
__global__ void __launch_bounds__(kSolveThreads, kSolveBlocks) early_solve_kernel(SolveArgs A) {
  __shared__ WarpShare s_share[kSolveThreads / 32];
  WarpShare& W = s_share[threadIdx.x >> 5];
  const uint32_t n = A.live[0], warps = gridDim.x * (kSolveThreads / 32u), lane = threadIdx.x & 31u;
  for (uint32_t j = (blockIdx.x * kSolveThreads + threadIdx.x) >> 5; j < n; j += warps) {
    const uint64_t k = A.first + A.live[1u + j];
    const uint32_t s = (uint32_t)(k / A.n_chains), c = (uint32_t)(k % A.n_chains);
    omg_mesh_record r;
    const omg_chain ch = A.chains[c];
    if (!mesh_record<WARP>(A.E, ch, A.ids[s], A.pos[3 * s], A.pos[3 * s + 1], A.pos[3 * s + 2], A.lx, A.ly, A.lz,
                           A.extras, A.n_extras, W, r))
      no_record(r, A.ids[s], ch);
    if (lane == 0) A.out[k] = r;
    __syncwarp();
  }
}

// Whole-warp closest hits (64 sources: 535 us a call, 617 us with the first lane
// of each warp alone; 512 sources 1541, 1953 us) need the split of every node (host-numbered trees,
// those with a 4-wide form) and the reference's triangle test.
bool warp_walks(const DEarly& E) {
  return (E.S.n_nodes4 != 0 || E.S.root < 0) && E.S.prims_wt == nullptr;
}

}  // namespace

cudaError_t launch_early_discover(const DEarly& E, const float lis[3], uint32_t n_rays, uint32_t rot, bool use_boxes,
                                  const float* jitter, unsigned long long* cand_key, omg_chain* cand_chain,
                                  uint32_t* cand_slot, unsigned long long* tkey, uint32_t* tidx, uint32_t tcap,
                                  omg_chain* out, uint32_t cap, uint32_t* n_out, cudaStream_t s) {
  DiscArgs A;
  A.E = E;
  A.lx = lis[0];
  A.ly = lis[1];
  A.lz = lis[2];
  A.n_rays = n_rays;
  A.rot = rot;
  A.use_boxes = use_boxes ? 1u : 0u;
  A.ga = 3.14159265358979323846f * (3.0f - sqrtf(5.0f));
  A.jitter = jitter;
  A.cand_key = cand_key;
  A.cand_chain = cand_chain;
  A.cand_slot = cand_slot;
  A.tkey = tkey;
  A.tidx = tidx;
  A.tcap = tcap;
  const uint32_t resident = E.n_sms * kDiscBlocks * (kDiscThreads / 32u);
  const bool warp = warp_walks(E) && n_rays <= 2u * resident;
  A.rays_per_warp = std::min(32u, std::max(1u, (n_rays + resident - 1u) / resident));
  const uint32_t per_block = (warp ? 1u : A.rays_per_warp) * (kDiscThreads / 32u);
  const uint32_t blocks = (n_rays + per_block - 1u) / per_block;
  if (n_rays && warp)
    early_discover_kernel<true><<<blocks, kDiscThreads, 0, s>>>(A);
  else if (n_rays)
    early_discover_kernel<false><<<blocks, kDiscThreads, 0, s>>>(A);
  early_compact_kernel<<<1, kCompactThreads, 0, s>>>(cand_key, cand_chain, cand_slot, tidx, 3u * n_rays, out, cap,
                                                     n_out);
  return cudaGetLastError();
}

cudaError_t launch_early_solve(const DEarly& E, const uint16_t* ids, const float* pos, uint32_t n_src,
                               const omg_chain* chains, uint32_t n_chains, const float lis[3], const omg_aabb* extras,
                               uint32_t n_extras, uint32_t* live, omg_mesh_record* out, cudaStream_t s) {
  SolveArgs A;
  A.E = E;
  A.ids = ids;
  A.pos = pos;
  A.n_src = n_src;
  A.chains = chains;
  A.n_chains = n_chains;
  A.lx = lis[0];
  A.ly = lis[1];
  A.lz = lis[2];
  A.extras = extras;
  A.n_extras = n_extras;
  A.live = live;
  A.out = out;
  const uint64_t n = (uint64_t)n_src * n_chains;
  if (n == 0) return cudaSuccess;
  for (A.first = 0; A.first < n; A.first += kEarlySlice) {
    A.n = (uint32_t)std::min<uint64_t>(kEarlySlice, n - A.first);
    const cudaError_t e = cudaMemsetAsync(live, 0, 4, s);
    if (e != cudaSuccess) return e;
    early_sift_kernel<<<(A.n + kSiftThreads - 1u) / kSiftThreads, kSiftThreads, 0, s>>>(A);
    const uint32_t blocks = std::min((A.n + kSolveThreads / 32u - 1u) / (kSolveThreads / 32u), E.n_sms * kSolveBlocks);
    if (warp_walks(E))
      early_solve_kernel<true><<<blocks, kSolveThreads, 0, s>>>(A);
    else
      early_solve_kernel<false><<<blocks, kSolveThreads, 0, s>>>(A);
  }
  return cudaGetLastError();
}

}  // namespace omg
