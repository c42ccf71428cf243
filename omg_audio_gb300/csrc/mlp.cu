// A tcgen05 GEMM of its own (omg_tc_gemm, omg_tc_gemm_bench), the accumulator
// in TMEM. (The surrogate's network runs whole passes a launch: mlp_net.cu.)
//
// GEMM: D[M x N] = A[M x K] . B[N x K]^T with A, B in BF16 and FP32
// accumulation. Operands are read through strides: element (m, k) of A is
// A[m a_rs + k a_ks]. One CTA of 128 threads computes a 128 x n_tile tile
// (n_tile <= 256) in 64-wide K chunks staged into shared memory as K-major
// core matrices (tc_gemm.cuh); one thread issues four K = 16 MMAs per chunk
// and commits them to an mbarrier (bounded waits). When both operands are
// K-major and 16-byte aligned, the chunks are staged by a three-deep cp.async
// pipeline, so the copies of the next chunks run under the current MMAs;
// otherwise each chunk is staged by plain loads. The epilogue reads the
// accumulator with tcgen05.ld and writes the rows through shared memory, whole
// lines at a time. A grid z dimension splits K; the split partials are added
// atomically.
#include <algorithm>

#include <cuda_bf16.h>

#include "omg_internal.h"
#include "tc_gemm.cuh"

namespace omg {

namespace {

constexpr uint32_t kTileM = 128;
constexpr uint32_t kMaxTileN = 256;
constexpr uint32_t kPolls = 1u << 24;   // mbarrier poll limit (error 16 in the error word)

// Stage rows [r0, r0 + rows) x K [k0, k0 + 64) of an operand into a tile.
__device__ __forceinline__ void stage(uint8_t* tile, const __nv_bfloat16* __restrict__ X, int64_t rs, int64_t ks,
                                      uint32_t r0, uint32_t rows, uint32_t R, uint32_t k0, uint32_t K) {
  const uint32_t pieces = rows * 8u;  // 16-byte pieces: (row, k8)
  for (uint32_t p = threadIdx.x; p < pieces; p += blockDim.x) {
    // consecutive threads take consecutive rows of the same k8 (coalesced when ks != 1)
    const uint32_t r = p % rows, k8 = p / rows;
    const uint32_t gr = r0 + r, gk = k0 + 8u * k8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (gr < R) {
      const __nv_bfloat16* src = X + (int64_t)gr * rs + (int64_t)gk * ks;
      if (ks == 1 && gk + 8u <= K && ((reinterpret_cast<uintptr_t>(src) & 15u) == 0u)) {
        v = *reinterpret_cast<const uint4*>(src);
      } else {
        uint16_t h[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          h[j] = 0;
          if (gk + (uint32_t)j < K) h[j] = __bfloat16_as_ushort(src[(int64_t)j * ks]);
        }
        v.x = (uint32_t)h[0] | ((uint32_t)h[1] << 16);
        v.y = (uint32_t)h[2] | ((uint32_t)h[3] << 16);
        v.z = (uint32_t)h[4] | ((uint32_t)h[5] << 16);
        v.w = (uint32_t)h[6] | ((uint32_t)h[7] << 16);
      }
    }
    *reinterpret_cast<uint4*>(tile + tc::tile_offset(r, 8u * k8)) = v;
  }
}

// Asynchronous staging of rows [r0, r0 + rows) x K [k0, k0 + 64) of a K-major
// operand (element (r, k) at X[r rs + k], rs a multiple of 8, X 16-byte
// aligned, K a multiple of 8): one 16-byte cp.async per (row, k8) piece,
// zero-filled beyond R rows or K.
__device__ __forceinline__ void stage_async(uint8_t* tile, const __nv_bfloat16* __restrict__ X, int64_t rs,
                                            uint32_t r0, uint32_t rows, uint32_t R, uint32_t k0, uint32_t K) {
  const uint32_t pieces = rows * 8u;
  for (uint32_t p = threadIdx.x; p < pieces; p += blockDim.x) {
    // 8 consecutive threads take the same k8 of 8 consecutive rows (their 128
    // bytes of shared memory are contiguous: no bank conflict); a warp reads 64
    // contiguous bytes of each of its 8 rows
    const uint32_t r = ((p >> 6) << 3) | (p & 7u), k8 = (p >> 3) & 7u;
    const uint32_t gr = r0 + r, gk = k0 + 8u * k8;
    const bool in = gr < R && gk < K;
    const __nv_bfloat16* src = in ? X + (int64_t)gr * rs + gk : X;
    tc::cp_async16(tile + tc::tile_offset(r, 8u * k8), src, in ? 16u : 0u);
  }
}

constexpr uint32_t kStages = 3;   // cp.async pipeline depth

// The epilogue. The accumulator comes out of TMEM one row per thread
// (tcgen05.ld 32x32b); each warp stages 32 x 32 blocks in shared memory (the
// operand stages, free once the last MMA has completed) and writes them row by
// row with consecutive lanes on consecutive columns: whole 128-byte lines
// instead of one sector per element.
__device__ __forceinline__ void gemm_epilogue(const GemmArgs& g, uint8_t* smem, uint32_t taddr, uint32_t m0,
                                              uint32_t n0, uint32_t nt, uint32_t nt16) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  float* st = reinterpret_cast<float*>(smem) + warp * (32u * 33u);
  const uint32_t lane_addr = taddr + ((warp * 32u) << 16);
  for (uint32_t c = 0; c < nt16; c += 32u) {
    const uint32_t w = min(32u, nt16 - c);               // 16 or 32 columns
    float a[16], b[16];
    tc::tmem_ld16(lane_addr + c, a);
    if (w == 32u) tc::tmem_ld16(lane_addr + c + 16u, b);
#pragma unroll
    for (uint32_t j = 0; j < 16u; j++) {
      st[lane * 33u + j] = a[j];
      if (w == 32u) st[lane * 33u + 16u + j] = b[j];
    }
    __syncwarp();
    const uint32_t col = n0 + c + lane;
    const bool ok = lane < w && c + lane < nt;
    for (uint32_t r = 0; r < 32u; r++) {
      const uint32_t row = m0 + warp * 32u + r;
      if (row >= g.M) break;
      if (!ok) continue;
      float* d = g.D + (int64_t)row * g.ldd + col;
      if (g.accumulate) atomicAdd(d, st[r * 33u + lane]);
      else *d = st[r * 33u + lane];
    }
    __syncwarp();
  }
}

// D = A . B^T on a 128 x n_tile tile. ASYNC: both operands K-major and
// 16-byte aligned, staged by a kStages-deep cp.async pipeline (the copies of
// the next chunks run under the MMAs of the current one); otherwise each
// 64-wide K chunk is staged by plain loads, then multiplied.
template <bool ASYNC>
__global__ void __launch_bounds__(128, 1) gemm_kernel(GemmArgs g) {
  const __nv_bfloat16* __restrict__ gA = static_cast<const __nv_bfloat16*>(g.A);
  const __nv_bfloat16* __restrict__ gB = static_cast<const __nv_bfloat16*>(g.B);
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t mbar[kStages];
  __shared__ uint32_t taddr_s;
  __shared__ uint32_t failed;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t m0 = blockIdx.x * kTileM;
  const uint32_t n0 = blockIdx.y * g.n_tile;
  const uint32_t nt = min(g.n_tile, g.N - n0);          // columns of this tile
  const uint32_t nt16 = (nt + 15u) & ~15u;              // MMA N (multiple of 16)
  const uint32_t stage_bytes = (kTileM + g.n_tile) * tc::kChunkK * 2u;
  // this CTA's K range
  const uint32_t k_per = ((g.K + gridDim.z - 1) / gridDim.z + tc::kChunkK - 1) / tc::kChunkK * tc::kChunkK;
  const uint32_t kb = blockIdx.z * k_per;
  const uint32_t ke = min(g.K, kb + k_per);
  const uint32_t nk = ke > kb ? (ke - kb + tc::kChunkK - 1) / tc::kChunkK : 0u;
  if (threadIdx.x == 0) {
    for (uint32_t i = 0; i < kStages; i++) tc::mbar_init(&mbar[i], 1);
    failed = 0;
  }
  // TMEM columns: the tile's width rounded up to a power of two (>= 32)
  uint32_t tcols = 32u;
  while (tcols < ((g.n_tile + 15u) & ~15u)) tcols <<= 1;
  if (warp == 0) tc::tmem_alloc(&taddr_s, tcols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = taddr_s;
  const uint32_t idesc = tc::idesc_bf16_f32(nt16, kTileM);
  uint32_t phase_bits = 0;   // bit b: the parity of buffer b's next completion
  uint32_t issued = 0;       // chunks whose MMAs have been issued (the same count in every thread)
  auto issue = [&](uint32_t buf, bool acc0) {
    uint8_t* sa = smem + buf * stage_bytes;
    uint8_t* sb = sa + kTileM * tc::kChunkK * 2u;
    tc::fence_after_sync();
    const uint32_t a0 = tc::smem_u32(sa), b0 = tc::smem_u32(sb);
#pragma unroll
    for (uint32_t s = 0; s < tc::kChunkK / 16u; s++)
      tc::mma_bf16(taddr, tc::smem_desc(a0 + 256u * s), tc::smem_desc(b0 + 256u * s), idesc, acc0 || s > 0);
    tc::mma_commit(&mbar[buf]);
  };
  auto wait_buf = [&](uint32_t buf) {
    if (!tc::mbar_wait(&mbar[buf], (phase_bits >> buf) & 1u, kPolls)) failed = 1;
    phase_bits ^= 1u << buf;
  };
  if (ASYNC) {
    auto load = [&](uint32_t chunk) {
      uint8_t* sa = smem + (chunk % kStages) * stage_bytes;
      uint8_t* sb = sa + kTileM * tc::kChunkK * 2u;
      const uint32_t k0 = kb + chunk * tc::kChunkK;
      stage_async(sa, gA, g.a_rs, m0, kTileM, g.M, k0, ke);
      stage_async(sb, gB, g.b_rs, n0, nt16, n0 + nt, k0, ke);
    };
    for (uint32_t c = 0; c + 1 < kStages; c++) {
      if (c < nk) load(c);
      tc::cp_async_commit();
    }
    for (uint32_t i = 0; i < nk; i++) {
      tc::cp_async_wait<kStages - 2>();     // chunk i has landed (this thread's copies)
      tc::fence_proxy_async();
      __syncthreads();                      // ... and every thread's
      if (threadIdx.x == 0) issue(i % kStages, i > 0);
      issued = i + 1;
      const uint32_t j = i + kStages - 1;   // refill the buffer chunk i - 1 used
      if (j < nk) {
        if (i >= 1) wait_buf((i - 1) % kStages);
        __syncthreads();
        if (failed) break;
        load(j);
      }
      tc::cp_async_commit();
    }
    tc::cp_async_wait_all();
  } else {
    uint8_t* sa = smem;
    uint8_t* sb = smem + kTileM * tc::kChunkK * 2u;
    for (uint32_t i = 0; i < nk; i++) {
      const uint32_t k0 = kb + i * tc::kChunkK;
      stage(sa, gA, g.a_rs, g.a_ks, m0, kTileM, g.M, k0, ke);
      stage(sb, gB, g.b_rs, g.b_ks, n0, nt16, n0 + nt, k0, ke);
      tc::fence_proxy_async();
      __syncthreads();
      if (threadIdx.x == 0) issue(0, i > 0);
      issued = i + 1;
      // the tiles are read asynchronously: wait before restaging them
      wait_buf(0);
      __syncthreads();
      if (failed) break;
    }
  }
  // the last chunk's MMAs (and with them, in order, every earlier one)
  if (ASYNC && !failed && nk > 0) wait_buf((nk - 1) % kStages);
  __syncthreads();
  tc::fence_after_sync();
  if (!failed && nk > 0) {
    gemm_epilogue(g, smem, taddr, m0, n0, nt, nt16);
  } else if (failed) {
    // give the last MMAs issued one more bounded wait before the TMEM is freed
    // (the slow path's only buffer was waited on already)
    if (ASYNC && issued > 0) {
      const uint32_t b = (issued - 1) % kStages;
      tc::mbar_wait(&mbar[b], (phase_bits >> b) & 1u, kPolls);
    }
    if (threadIdx.x == 0 && g.err) atomicOr(g.err, 16u);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, tcols);
}

}  // namespace

size_t gemm_smem_bytes() { return (size_t)(kTileM + kMaxTileN) * tc::kChunkK * 2; }

namespace {
bool k_major_ok(const void* p, int64_t rs, int64_t ks) {
  return ks == 1 && rs % 8 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}
}  // namespace

namespace {
constexpr int kMaxDev = 64;
bool g_attr_done[kMaxDev] = {};
}  // namespace

// The GEMM kernels' shared-memory limits, once per device (call it outside
// any stream capture, before the first launch_gemm on a device).
cudaError_t gemm_init() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  if (g_attr_done[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem_bytes());
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kStages * gemm_smem_bytes()));
  if (e != cudaSuccess) return e;
  g_attr_done[dev] = true;
  return cudaSuccess;
}

cudaError_t launch_gemm(const GemmArgs& g, uint32_t k_split, cudaStream_t s) {
  if (g.M == 0 || g.N == 0 || g.K == 0) return cudaSuccess;
  if (g.n_tile == 0 || g.n_tile > kMaxTileN || (g.n_tile & 15u)) return cudaErrorInvalidValue;
  cudaError_t e = gemm_init();
  if (e != cudaSuccess) return e;
  dim3 grid((g.M + kTileM - 1) / kTileM, (g.N + g.n_tile - 1) / g.n_tile, k_split ? k_split : 1);
  const size_t stage = (size_t)(kTileM + g.n_tile) * tc::kChunkK * 2;
  if (k_major_ok(g.A, g.a_rs, g.a_ks) && k_major_ok(g.B, g.b_rs, g.b_ks) && g.K % 8 == 0)
    gemm_kernel<true><<<grid, 128, kStages * stage, s>>>(g);
  else
    gemm_kernel<false><<<grid, 128, stage, s>>>(g);
  return cudaGetLastError();
}

}  // namespace omg
