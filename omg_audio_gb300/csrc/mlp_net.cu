// The surrogate's network on the tensor cores, whole passes a launch:
//   rows_kernel    one CTA takes 128 rows of one member through every layer:
//                  inference, or the forward pass, the loss and the backward
//                  chain of a training step
//   dw_kernel      the weight gradients of every layer and member
//   adamw_kernel   the optimizer over every parameter
//   ensemble_kernel  the members' mean and spread
//
// What bounds it, and why whole passes. A layer is 0.5 GFLOP for the training
// batch (0.3 us of the chip), so a launch per layer spends its time in launch
// gaps, prologues and trips of the activations through L2: 22 dependent launches
// of 6 to 34 us made a training step of the 38-256x4-192 ensemble at 4096 rows
// 583 us. Rows do not meet before the weight gradients, so a CTA keeps its rows'
// activations in shared memory from the first layer to the last and back, and
// only the weights stream in, one 128 KB layer ahead, while the previous
// layer's epilogue runs. The epilogues (bias, GELU and its derivative from one
// tanh, per element) are then the largest part: 16 warps share them.
//
// Operand images. An activation tile (128 rows) and a layer's weights are kept,
// in shared and in global memory alike, as 8 x 8 core matrices (128 B: 8 rows of
// 8 consecutive features), the row groups of one feature block contiguous:
//   element (row, k): (k / 8) * 16 R + 16 row + 2 (k % 8) bytes, R rows
// One bulk copy moves a whole tile or layer. Read K-major the image is the
// operand of the forward product (and dZ of the input gradient); read MN-major
// it is the transposed operand of the weight gradient (both sides) and of the
// input gradient (the weights), so nothing is transposed in memory.
#include <algorithm>
#include <utility>

#include <cuda_bf16.h>

#include "mlp_net.h"
#include "tc_gemm.cuh"

namespace omg {

namespace {

constexpr uint32_t kRows = 128;               // rows a CTA owns (the MMA's M)
constexpr uint32_t kWide = kMlpWide;          // widest layer, and the first layer's K a step
constexpr uint32_t kRowThreads = 512;
constexpr uint32_t kTileBytes = kRows * kWide * 2;
constexpr uint32_t kWBytes = kWide * kWide * 2;
constexpr uint32_t kSumFloats = 32u * 16u;    // column_sum16's scratch, a warp
template <bool TRAIN>
constexpr uint32_t kRowsSmem = kTileBytes + kWBytes + (TRAIN ? kRowThreads / 32u * kSumFloats * 4u : 0u);
constexpr uint32_t kPolls = 1u << 22;         // mbarrier poll limit (error 16 in the error word)

__device__ __forceinline__ float gelu_f(float z, float t) { return 0.5f * z * (1.0f + t); }

// tanh form of GELU: the inner tanh, shared by the value and the derivative
__device__ __forceinline__ float gelu_tanh(float z) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = k0 * (z + k1 * z * z * z);
  return tanhf(u);
}

__device__ __forceinline__ float gelu_grad(float z, float t) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float du = k0 * (1.0f + 3.0f * k1 * z * z);
  return 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * du;
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);   // one conversion, a in the low half
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 16 consecutive features of one row into the tile image, and into its copy in
// global memory where there is one (two 16-byte stores each; a warp's lanes are
// consecutive rows: contiguous, no bank conflict). The copies are the weight
// gradients' operands. (A bulk store of the finished tile reads it at the rate at
// which all blocks' bursts drain, and the next epilogue waited for that before it
// overwrote the tile, 2800 cycles a layer: 64 training steps 7.63 -> 7.58 ms, with
// the last hidden layer's GELU' in TMEM 7.49.)
__device__ __forceinline__ void put16(uint8_t* tile, uint8_t* copy, uint32_t row, uint32_t c, const float (&v)[16]) {
  const uint32_t at = (c >> 3) * (16u * kRows) + 16u * row;
  const uint4 a = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7])),
              b = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
  *reinterpret_cast<uint4*>(tile + at) = a;
  *reinterpret_cast<uint4*>(tile + at + 16u * kRows) = b;
  if (copy) {
    *reinterpret_cast<uint4*>(copy + at) = a;
    *reinterpret_cast<uint4*>(copy + at + 16u * kRows) = b;
  }
}

// Sums of 16 columns over the warp's 32 rows: row r, r + 8, r + 16, r + 24 one after
// another for r = 0 .. 7, then those eight in order (a bias gradient's rounding moves
// whole AdamW steps where the gradient is near zero, so the order stays what it was).
// Through 2 KB of shared memory, a lane per half column: a row lies at 16 h + 4 k + i
// (r = 8 k + 4 h + i), turned by its column, so neither the stores nor the loads
// conflict. Lanes below 16 return their column's sum. (A halving tree of 16 shuffles
// added in another order: rows_kernel 70.0 us for a training step of 4 x 38-256x4-192
// at 4096 rows, 75.4 this way.)
__device__ __forceinline__ float column_sum16(float* __restrict__ w, const float (&v)[16], uint32_t lane) {
  const uint32_t p = ((lane & 4u) << 2) | ((lane >> 1) & 12u) | (lane & 3u);
#pragma unroll
  for (uint32_t j = 0; j < 16; j++) w[32u * j + ((p + j) & 31u)] = v[j];
  __syncwarp();
  const uint32_t c = lane & 15u, at = (lane & 16u) + c;
  float part[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) {
    part[i] = w[32u * c + ((at + i) & 31u)];
#pragma unroll
    for (uint32_t k = 1; k < 4; k++) part[i] += w[32u * c + ((at + 4u * k + i) & 31u)];
  }
  __syncwarp();   // read before the next columns are stored
  float t = part[0] + part[1];
  t += part[2];
  t += part[3];
#pragma unroll
  for (int i = 0; i < 4; i++) t += __shfl_down_sync(0xffffffffu, part[i], 16);
  return t;
}

// The accumulator's columns [lo, hi) in chunks of 16 through f(column, values):
// the next chunk is on its way out of TMEM while this one is worked on.
template <class F>
__device__ __forceinline__ void for_columns(uint32_t lanes, uint32_t lo, uint32_t hi, F&& f) {
  if (lo >= hi) return;
  float a[16], b[16];
  tc::tmem_ld16_async(lanes + lo, a);
  for (uint32_t c = lo;;) {
    tc::tmem_wait(a);
    if (c + 16u < hi) tc::tmem_ld16_async(lanes + c + 16u, b);
    f(c, a);
    c += 16u;
    if (c >= hi) break;
    tc::tmem_wait(b);
    if (c + 16u < hi) tc::tmem_ld16_async(lanes + c + 16u, a);
    f(c, b);
    c += 16u;
    if (c >= hi) break;
  }
}

// TMEM: the accumulator, and in training GELU' of the last hidden layer beside it
// (one block a multiprocessor: the other half is free); the other hidden layers'
// goes through global memory.
template <bool TRAIN>
constexpr uint32_t kRowsTmem = TRAIN ? 2u * kWide : kWide;

template <bool TRAIN>
__global__ void __launch_bounds__(kRowThreads, 1) rows_kernel(const __grid_constant__ MlpRowsArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* tile = smem;                        // the rows' activations (or gradients) of the current layer
  uint8_t* wbuf = smem + kTileBytes;           // the current layer's weights
  float* sums = reinterpret_cast<float*>(wbuf + kWBytes) + (threadIdx.x >> 5) * kSumFloats;   // (training only)
  __shared__ __align__(8) uint64_t bar_w, bar_mma;
  __shared__ uint32_t taddr_s;
  __shared__ float s_bias[kWide];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t row = (warp & 3u) * 32u + lane, cg = warp >> 2;   // TMEM lane, column group (4 of them)
  const uint32_t t0 = blockIdx.x, member = g.member0 + blockIdx.y;
  const MlpNet& N = g.net;
  const uint32_t L = N.n_layers;
  const float* P = g.P + (uint64_t)member * N.p_stride;
  const uint16_t* img = g.img + (uint64_t)member * N.img_stride;
  const uint32_t grow = t0 * kRows + row;      // this thread's row of the batch
  const bool live = t0 * kRows + (warp & 3u) * 32u < g.rows;       // (warp-uniform) any row of the warp
  if (tid == 0) {
    tc::mbar_init(&bar_w, 1);
    tc::mbar_init(&bar_mma, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(&taddr_s, kRowsTmem<TRAIN>);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = taddr_s;
  const uint32_t my_lanes = taddr + (((warp & 3u) * 32u) << 16);
  uint32_t par_w = 0, par_mma = 0;             // thread 0's and every thread's next phase
  bool loading = false;                        // thread 0: a weight load is in flight
  bool ok = true;

  // weights of layer l, K chunk c of kWide features (thread 0)
  auto load_w = [&](uint32_t l, uint32_t c) {
    const MlpLayerDesc& D = N.L[l];
    const uint32_t k0 = c * kWide, kn = min(kWide, D.ip - k0), bytes = kn * D.op * 2u;
    tc::mbar_expect_tx(&bar_w, bytes);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(img + D.img_off) + (uint64_t)k0 * D.op * 2u;
    for (uint32_t o = 0; o < bytes; o += 32768u) tc::bulk_load(wbuf + o, src + o, min(32768u, bytes - o), &bar_w);
    loading = true;
  };
  auto wait_w = [&]() {
    if (!loading) return;
    if (!tc::mbar_wait(&bar_w, par_w, kPolls)) {
      ok = false;                              // still in flight: the block's end waits for it again
      return;
    }
    par_w ^= 1u;
    loading = false;
  };
  // the tile (K features) times the weights read K-major (bwd = false: N = op)
  // or MN-major (bwd: N = ip), accumulated over K; the commit arrives on bar_mma
  auto issue = [&](const MlpLayerDesc& D, bool bwd, uint32_t kn, bool acc0) {
    tc::fence_after_sync();
    const uint32_t a0 = tc::smem_u32(tile), b0 = tc::smem_u32(wbuf);
    const uint32_t lead = 16u * D.op;          // bytes between the image's feature blocks
    const uint32_t idesc = tc::idesc_bf16_f32(bwd ? D.ip : D.op, kRows) | (bwd ? tc::kTransB : 0u);
    for (uint32_t s = 0; s < kn / 16u; s++) {
      const uint64_t ad = tc::smem_desc(a0 + s * (32u * kRows), 16u * kRows, 128u);
      const uint64_t bd = bwd ? tc::smem_desc(b0 + 256u * s, 128u, lead) : tc::smem_desc(b0 + s * 2u * lead, lead, 128u);
      tc::mma_bf16(taddr, ad, bd, idesc, acc0 || s > 0);
    }
    tc::mma_commit(&bar_mma);
  };
  auto wait_mma = [&]() {
    ok = tc::mbar_wait(&bar_mma, par_mma, kPolls) && ok;
    par_mma ^= 1u;
  };
  // the columns of a layer of width w that this thread's warp handles
  auto col_lo = [&](uint32_t w) { return min(w, cg * (((w >> 4) + 3u) / 4u) * 16u); };
  auto col_hi = [&](uint32_t w) { return min(w, (cg + 1u) * (((w >> 4) + 3u) / 4u) * 16u); };

  tc::grid_wait();
  const uint64_t mt = (uint64_t)blockIdx.y * gridDim.x + t0;       // this CTA's slot of the scratch arrays
  float* gb = TRAIN ? g.gb + (mt * (kRows / 32u) + (warp & 3u)) * L * kWide : nullptr;   // these 32 rows' bias sums
  const uint32_t* idx = nullptr;
  uint64_t src_row = grow;
  if (TRAIN && g.perm) {
    const uint32_t step = *g.step;
    idx = g.perm + (uint64_t)((step / g.spe) & 1u) * g.perm_half + (uint64_t)member * g.perm_member +
          (uint64_t)(step % g.spe) * g.rows;
    src_row = idx[grow];
  }
  if (tid == 0) load_w(0, 0);

  // ---------------------------------------------------------------- forward
  for (uint32_t l = 0; l < L; l++) {
    const MlpLayerDesc& D = N.L[l];
    const uint32_t chunks = (D.ip + kWide - 1) / kWide;            // 1 beyond the first layer
    for (uint32_t c = 0; c < chunks; c++) {
      const uint32_t k0 = c * kWide, kn = min(kWide, D.ip - k0);
      if (l == 0 && live) {
        // inputs (standardized here for inference) to bf16, eight features a store
        for (uint32_t f = 8u * cg; f < kn; f += 32u) {
          float v[8];
#pragma unroll
          for (uint32_t j = 0; j < 8; j++) {
            const uint32_t k = k0 + f + j;
            v[j] = 0.0f;
            if (k < D.in && grow < g.rows) {
              v[j] = g.X[src_row * D.in + k];
              if (!TRAIN) v[j] = (v[j] - g.x_mean[k]) / g.x_sd[k];
            }
          }
          const uint32_t at = (f >> 3) * (16u * kRows) + 16u * row;
          const uint4 w = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
          *reinterpret_cast<uint4*>(tile + at) = w;
          if (TRAIN)
            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(g.xt + mt * (kRows * D.ip) + (uint64_t)k0 * kRows) + at) = w;
        }
      }
      tc::fence_proxy_async();
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        wait_w();
        if (ok) issue(D, false, kn, c > 0);
      }
      if (ok) wait_mma();
      if (tid == 0) {
        // the weight buffer is free: the next chunk or layer under this epilogue
        if (c + 1 < chunks) load_w(l, c + 1);
        else if (l + 1 < L) load_w(l + 1, 0);
      }
      if (c + 1 == chunks)
        for (uint32_t i = tid; i < D.op; i += kRowThreads) s_bias[i] = i < D.out ? P[D.b_off + i] : 0.0f;
      if (__syncthreads_or(!ok)) goto bail;
      tc::fence_after_sync();
    }
    if (l + 1 < L) {
      if (live) {
        uint8_t* copy = TRAIN ? reinterpret_cast<uint8_t*>(g.at + (mt * (L - 1u) + l) * (kRows * D.op)) : nullptr;
        for_columns(my_lanes, col_lo(D.op), col_hi(D.op), [&](uint32_t c, float (&v)[16]) {
          float gp[16];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const float z = v[j] + s_bias[c + j];
            const float t = gelu_tanh(z);
            v[j] = gelu_f(z, t);
            if (TRAIN) gp[j] = gelu_grad(z, t);
          }
          put16(tile, copy, row, c, v);
          if (TRAIN && l + 2 == L) {
            tc::tmem_st16(my_lanes + kWide + c, gp);
          } else if (TRAIN) {
            // GELU'(z) in f32 for the way back, read again by this thread alone
            float4* gd = reinterpret_cast<float4*>(g.gz) + ((mt * (L - 1u) + l) * (D.op / 4u) + c / 4u) * kRows + row;
#pragma unroll
            for (int q = 0; q < 4; q++)
              gd[q * kRows] = make_float4(gp[4 * q], gp[4 * q + 1], gp[4 * q + 2], gp[4 * q + 3]);
          }
        });
      }
    } else if (!TRAIN) {
      float* o = g.out + ((uint64_t)blockIdx.y * g.rows + grow) * D.out;
      if (live) {
        for_columns(my_lanes, col_lo(D.op), col_hi(D.op), [&](uint32_t c, float (&v)[16]) {
          if (grow < g.rows) {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] += s_bias[c + j];
            if (D.out % 4u == 0u && c + 16u <= D.out) {
#pragma unroll
              for (int q = 0; q < 4; q++)
                reinterpret_cast<float4*>(o + c)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 16; j++)
                if (c + j < D.out) o[c + j] = v[j];
            }
          }
        });
      }
    } else {
      // the mean squared error and its gradient
      const float inv_n = 1.0f / ((float)g.rows * (float)D.out);
      const uint32_t lo = col_lo(D.op), hi = col_hi(D.op);
      uint8_t* copy = reinterpret_cast<uint8_t*>(g.dzt + (mt * L + l) * (kRows * kWide));
      float lsum = 0.0f;
      float y[16];
      const float* yr = g.Y + src_row * D.out;
      auto load_y = [&](uint32_t c) {
        if (D.out % 4u == 0u) {
          const float4* y4 = reinterpret_cast<const float4*>(yr + c);
#pragma unroll
          for (uint32_t q = 0; q < 4; q++) {
            const float4 w = c + 4u * q < D.out ? __ldg(y4 + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            y[4 * q] = w.x;
            y[4 * q + 1] = w.y;
            y[4 * q + 2] = w.z;
            y[4 * q + 3] = w.w;
          }
        } else {
#pragma unroll
          for (uint32_t j = 0; j < 16; j++) y[j] = c + j < D.out ? __ldg(yr + c + j) : 0.0f;
        }
      };
      if (lo < hi) load_y(lo);
      for_columns(my_lanes, lo, hi, [&](uint32_t c, float (&v)[16]) {
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const float e = c + j < D.out ? v[j] + s_bias[c + j] - y[j] : 0.0f;
          lsum += e * e;
          v[j] = 2.0f * e * inv_n;
        }
        if (c + 16u < hi) load_y(c + 16u);
        put16(tile, copy, row, c, v);
        const float s = column_sum16(sums, v, lane);
        if (lane < 16u) gb[l * kWide + c + lane] = s;
      });
      for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      if (lane == 0) atomicAdd(g.loss + member, lsum * inv_n);
    }
  }
  // --------------------------------------------------------------- backward
  if (TRAIN) {
    for (uint32_t l = L - 1;; l--) {
      const MlpLayerDesc& D = N.L[l];
      tc::fence_proxy_async();
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0 && l > 0) {
        wait_w();
        if (ok) issue(D, true, D.op, false);
      }
      if (l == 0) break;
      // dZ of the layer below = dX * GELU'(Z)
      const uint32_t lo = col_lo(D.ip), hi = col_hi(D.ip);
      const float4* gd = reinterpret_cast<const float4*>(g.gz) + (mt * (L - 1u) + (l - 1u)) * (D.ip / 4u) * kRows + row;
      uint8_t* copy = reinterpret_cast<uint8_t*>(g.dzt + (mt * L + (l - 1u)) * (kRows * kWide));
      // GELU'(z) of the next columns is loaded ahead: the first ones while the product runs
      float4 gp[4];
      auto load_g = [&](uint32_t c) {
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) gp[q] = gd[(c / 4u + q) * kRows];
      };
      const bool top = l + 1 == L;             // GELU' is in TMEM
      if (lo < hi && !top) load_g(lo);
      if (ok) wait_mma();
      if (tid == 0 && l > 1) load_w(l - 1, 0);
      if (__syncthreads_or(!ok)) goto bail;
      tc::fence_after_sync();
      for_columns(my_lanes, lo, hi, [&](uint32_t c, float (&v)[16]) {
        if (top) {
          float t[16];
          tc::tmem_ld16(my_lanes + kWide + c, t);
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] *= t[j];
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            v[4 * q] *= gp[q].x;
            v[4 * q + 1] *= gp[q].y;
            v[4 * q + 2] *= gp[q].z;
            v[4 * q + 3] *= gp[q].w;
          }
          if (c + 16u < hi) load_g(c + 16u);
        }
        put16(tile, copy, row, c, v);
        const float s = column_sum16(sums, v, lane);
        if (lane < 16u) gb[(l - 1u) * kWide + c + lane] = s;
      });
    }
  }
bail:
  if (!ok && g.err) atomicOr(g.err, 16u);
  if (tid == 0) {
    // what is still in flight (only after a wait ran out) ends before the block does
    if (loading) tc::mbar_wait(&bar_w, par_w, kPolls);
    if (!ok) tc::mbar_wait(&bar_mma, par_mma ^ 1u, kPolls);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, kRowsTmem<TRAIN>);
}

// The weight gradients: dW[out x in] = dZ^T A over the batch's rows, both read
// MN-major from the tile images that rows_kernel left. The rows are summed in
// shares (dw_shares), each a chain of MMAs into TMEM columns of its own. A CTA
// takes 128 output features x up to 256 input features of one layer of one member
// over consecutive shares, two row tiles in flight (96 KB each), adds its shares
// up in their order and the result to the gradient; those with a layer's first share
// also add the rows' bias sums in order (one store a feature: no atomic's arrival
// order, so batches of up to two shares train to the same weights each time). Bound
// by the tiles' loads: 96 KB each for 1024 cycles of MMA. 26.9 us for the training step
// of 4 x 38-256x4-192 at 4096 rows, of 8 tiles a CTA; 25.1 us when the shares were cut
// to fill the chip and the biases added by rows_kernel's atomics.
constexpr uint32_t kDwThreads = 256;
constexpr uint32_t kDwA = 16u * 16u * kRows;          // dZ: 16 feature blocks
constexpr uint32_t kDwStage = kDwA + kTileBytes;
constexpr uint32_t kDwSmem = 2u * kDwStage;
constexpr uint32_t kDwTmem = 512;                     // one block a multiprocessor (its shared memory)
// TMEM columns of one share's accumulator, nn columns wide
__host__ __device__ __forceinline__ uint32_t dw_columns(uint32_t nn) {
  uint32_t c = 32;
  while (c < nn) c <<= 1;
  return c;
}

__global__ void __launch_bounds__(kDwThreads, 1) dw_kernel(const __grid_constant__ MlpDwArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) uint64_t full[2], done[2];
  __shared__ uint32_t taddr_s;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const MlpNet& N = g.net;
  const uint32_t L = N.n_layers;
  // this CTA's layer (widest first), member, feature block, input block, group of shares
  uint32_t u = blockIdx.x, l = 0, mh = 1, nh = 1, per = 1, groups = 1;
  for (uint32_t k = 0; k < L; k++) {
    l = k + 1 < L ? k + 1 : 0;
    mh = (N.L[l].op + 127u) / 128u;
    nh = (N.L[l].ip + kWide - 1) / kWide;
    per = l == 0 ? g.group0 : g.group;
    groups = (g.shares + per - 1) / per;
    const uint32_t units = mh * nh * g.members * groups;
    if (u < units) break;
    u -= units;
  }
  const MlpLayerDesc& D = N.L[l];
  const uint32_t h = (u / groups) % mh, nb = (u / groups / mh) % nh;
  const uint32_t mi = u / (groups * mh * nh);                         // member of this launch
  const uint32_t s0 = (u % groups) * per, ns = min(per, g.shares - s0);
  const uint32_t rb = s0 * g.share_rows, re = min(g.tiles * kRows, rb + ns * g.share_rows);   // its rows
  const uint32_t tb = rb / kRows, te = (re + kRows - 1) / kRows;      // (a share may end in the middle of a tile)
  const uint32_t n0 = nb * kWide, nn = min(kWide, D.ip - n0);
  const uint32_t mo = min(128u, D.op - 128u * h);                     // output features here (the rest of M is unused)
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&done[i], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc(&taddr_s, kDwTmem);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  tc::grid_wait();
  const uint32_t taddr = taddr_s;
  const uint32_t bz = mo * kRows * 2u, ba = nn * kRows * 2u, cols = dw_columns(nn);
  bool ok = true;
  const uint32_t n = te - tb;
  if (tid == 0) {
    auto load = [&](uint32_t i) {
      const uint64_t mt = (uint64_t)mi * g.tiles + tb + i;
      uint8_t* s = smem + (i & 1u) * kDwStage;
      const uint8_t* z = reinterpret_cast<const uint8_t*>(g.dzt + (mt * L + l) * (kRows * kWide)) + h * kDwA;
      const uint8_t* a = reinterpret_cast<const uint8_t*>(l == 0 ? g.xt + mt * (kRows * D.ip) + (uint64_t)n0 * kRows
                                                                 : g.at + (mt * (L - 1u) + (l - 1u)) * (kRows * D.ip));
      tc::mbar_expect_tx(&full[i & 1u], bz + ba);
      tc::bulk_load(s, z, bz, &full[i & 1u]);
      for (uint32_t o = 0; o < ba; o += 32768u)
        tc::bulk_load(s + kDwA + o, a + o, min(32768u, ba - o), &full[i & 1u]);
    };
    load(0);
    if (n > 1) load(1);
    const uint32_t idesc = tc::idesc_bf16_f32(nn, 128u) | tc::kTransA | tc::kTransB;
    uint32_t acc = taddr, in = 0;               // the share's columns, and its rows so far
    uint32_t loaded = min(2u, n), issued = 0;   // tiles under way
    for (uint32_t i = 0; i < n && ok; i++) {
      const uint32_t b = i & 1u, ph = (i >> 1) & 1u;
      ok = tc::mbar_wait(&full[b], ph, kPolls);
      if (!ok) break;
      const uint32_t a0 = tc::smem_u32(smem + b * kDwStage), b0 = a0 + kDwA;
      // the tile's rows of these shares, 16 a step
      const uint32_t r0 = (tb + i) * kRows, first = (max(rb, r0) - r0) / 16u, last = (min(re, r0 + kRows) - r0) / 16u;
      for (uint32_t s = first; s < last; s++) {
        tc::mma_bf16(acc, tc::smem_desc(a0 + 256u * s, 128u, 16u * kRows),
                     tc::smem_desc(b0 + 256u * s, 128u, 16u * kRows), idesc, in != 0u);
        in += 16u;
        if (in == g.share_rows) {
          in = 0;
          acc += cols;
        }
      }
      tc::mma_commit(&done[b]);
      issued = i + 1;
      // the stage is refilled once its MMAs are done, while the other stage's run
      if (i >= 1 && i + 1 < n) {
        ok = tc::mbar_wait(&done[b ^ 1u], ((i - 1) >> 1) & 1u, kPolls);
        if (ok) {
          load(i + 1);
          loaded = i + 2;
        }
      }
    }
    // the last MMAs (and with them every earlier one)
    if (ok) ok = tc::mbar_wait(&done[(n - 1) & 1u], ((n - 1) >> 1) & 1u, kPolls);
    if (!ok) {
      if (g.err) atomicOr(g.err, 16u);
      // one more bounded wait for what may be in flight: the last two loads, and the
      // last MMAs issued (with them every earlier one)
      for (uint32_t i = loaded > 2u ? loaded - 2u : 0u; i < loaded; i++) tc::mbar_wait(&full[i & 1u], (i >> 1) & 1u, kPolls);
      if (issued) tc::mbar_wait(&done[(issued - 1u) & 1u], ((issued - 1u) >> 1) & 1u, kPolls);
    }
  }
  // the bias gradients of these features: their sums of 32 rows in order, while the products run
  if (nb == 0 && s0 == 0 && tid >= kDwThreads - 128u) {
    const uint32_t o = 128u * h + (tid & 127u);
    if (o < D.out) {
      constexpr uint32_t kAhead = 16;
      const uint32_t groups32 = g.tiles * (kRows / 32u);          // a multiple of 4
      const float* b = g.gb + ((uint64_t)mi * groups32 * L + l) * kWide + o;
      float sum = 0.0f, v[kAhead];
      for (uint32_t q = 0; q < groups32; q += kAhead) {
#pragma unroll
        for (uint32_t j = 0; j < kAhead; j++) v[j] = q + j < groups32 ? b[(uint64_t)(q + j) * L * kWide] : 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < kAhead; j++) sum += v[j];
      }
      g.G[(uint64_t)(g.member0 + mi) * N.p_stride + D.b_off + o] = sum;
    }
  }
  if (!__syncthreads_or(!ok)) {
    tc::fence_after_sync();
    const uint32_t o = 128u * h + (warp & 3u) * 32u + lane;
    float* W = g.G + (uint64_t)(g.member0 + mi) * N.p_stride + D.w_off + (uint64_t)o * D.in + n0;
    const bool v4 = D.in % 4u == 0u;            // (w_off and n0 are multiples of 4)
    const uint32_t nv = min(nn, D.in - n0);     // columns that exist
    for (uint32_t c = 16u * (warp >> 2); c < nn; c += 32u) {
      float v[16];
      tc::tmem_ld16(taddr + (((warp & 3u) * 32u) << 16) + c, v);
      for (uint32_t q = 1; q < ns; q++) {
        float t[16];
        tc::tmem_ld16(taddr + (((warp & 3u) * 32u) << 16) + q * cols + c, t);
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] += t[j];
      }
      if (o < D.out) {
#pragma unroll
        for (uint32_t q = 0; q < 16; q += 4) {
          if (v4 && c + q < nv) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(W + c + q), "f"(v[q]), "f"(v[q + 1]),
                         "f"(v[q + 2]), "f"(v[q + 3])
                         : "memory");
          } else {
#pragma unroll
            for (uint32_t j = 0; j < 4; j++)
              if (c + q + j < nv) atomicAdd(W + c + q + j, v[q + j]);
          }
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, kDwTmem);
}

// bf16 copy of one parameter into its layer's image
__device__ __forceinline__ void put_image(uint16_t* img, const MlpLayerDesc& D, uint32_t o, uint32_t k, float x) {
  img[D.img_off + (uint64_t)(k >> 3) * (8u * D.op) + 8u * o + (k & 7u)] = __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// AdamW over every member's parameters, four a thread; the weights' bf16 images
// follow, and the gradients are left zero for the next step. The block that
// ends last closes the step: the counter, and at an epoch's end its losses.
__global__ void __launch_bounds__(256) adamw_kernel(const __grid_constant__ MlpAdamwArgs g) {
  const MlpNet& N = g.net;
  tc::grid_wait();
  const uint32_t t = *g.step, e = blockIdx.y;
  const float lr = g.sched[3u * t], bc1 = g.sched[3u * t + 1u], bc2 = g.sched[3u * t + 2u];
  const uint32_t p = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
  if (p < N.p_stride) {
    const uint64_t at = (uint64_t)e * N.p_stride + p;
    uint32_t l = 0;
    while (l + 1 < N.n_layers && p >= N.L[l + 1].w_off) l++;
    const MlpLayerDesc& D = N.L[l];
    const bool isw = p < D.b_off;               // (b_off is a multiple of 4: a quad is all weights or none)
    float4 W = reinterpret_cast<const float4*>(g.P)[at / 4];
    float4 M = reinterpret_cast<const float4*>(g.M1)[at / 4];
    float4 V = reinterpret_cast<const float4*>(g.V1)[at / 4];
    const float4 G = reinterpret_cast<const float4*>(g.G)[at / 4];
    float x[4] = {W.x, W.y, W.z, W.w}, m[4] = {M.x, M.y, M.z, M.w}, v[4] = {V.x, V.y, V.z, V.w};
    const float gr[4] = {G.x, G.y, G.z, G.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      m[j] = g.b1 * m[j] + (1.0f - g.b1) * gr[j];
      v[j] = g.b2 * v[j] + (1.0f - g.b2) * gr[j] * gr[j];
      const float mh = m[j] / bc1, vh = v[j] / bc2;
      x[j] = x[j] - lr * (mh / (sqrtf(vh) + g.eps) + (isw ? g.wd : 0.0f) * x[j]);
    }
    reinterpret_cast<float4*>(g.P)[at / 4] = make_float4(x[0], x[1], x[2], x[3]);
    reinterpret_cast<float4*>(g.M1)[at / 4] = make_float4(m[0], m[1], m[2], m[3]);
    reinterpret_cast<float4*>(g.V1)[at / 4] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(g.G)[at / 4] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (isw) {
      uint16_t* im = g.img + (uint64_t)e * N.img_stride;
      uint32_t i = p - D.w_off, o = i / D.in, k = i - o * D.in;
      if (D.in % 4u == 0u) {                    // the quad is one row's, half a core matrix row
        if (o < D.out)
          *reinterpret_cast<uint2*>(im + D.img_off + (uint64_t)(k >> 3) * (8u * D.op) + 8u * o + (k & 7u)) =
              make_uint2(pack2(x[0], x[1]), pack2(x[2], x[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (o < D.out) put_image(im, D, o, k, x[j]);
          if (++k == D.in) {
            k = 0;
            o++;
          }
        }
      }
    }
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(g.ticket, 1u) + 1u == gridDim.x * gridDim.y;
  }
  __syncthreads();
  if (last) {
    const bool ends = (t + 1u) % g.spe == 0u;
    if (threadIdx.x < N.members) {
      if (ends) g.epoch_loss[(uint64_t)threadIdx.x * g.epochs + t / g.spe] = g.loss[threadIdx.x];
      g.loss[threadIdx.x] = 0.0f;
    }
    if (threadIdx.x == 0) {
      *g.ticket = 0;
      *g.step = t + 1u;
    }
  }
}

// Every member's images from its f32 parameters
__global__ void image_kernel(const __grid_constant__ MlpNet N, const float* __restrict__ P, uint16_t* __restrict__ img) {
  const uint32_t e = blockIdx.y;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < N.p_stride; p += gridDim.x * blockDim.x) {
    uint32_t l = 0;
    while (l + 1 < N.n_layers && p >= N.L[l + 1].w_off) l++;
    const MlpLayerDesc& D = N.L[l];
    const uint32_t i = p - D.w_off;
    if (i < D.in * D.out)
      put_image(img + (uint64_t)e * N.img_stride, D, i / D.in, i % D.in, P[(uint64_t)e * N.p_stride + p]);
  }
}

// One warp per row: the members' outputs in the targets' units, their mean and
// spread (sums in member order), and per row the largest spread among outputs
// whose mean is >= level.
__global__ void __launch_bounds__(256) ensemble_kernel(const float* __restrict__ y, uint32_t members, uint32_t rows, uint32_t cols,
                                const float* __restrict__ mean, const float* __restrict__ sd, float inv_e,
                                float level, float* __restrict__ out_mean, float* __restrict__ out_std,
                                float* __restrict__ out_spread) {
  const uint32_t row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  tc::grid_wait();
  if (row >= rows) return;
  float most = 0.0f;
  for (uint32_t c = lane; c < cols; c += 32) {
    const float s = sd[c], b = mean[c];
    float a = 0.0f, a2 = 0.0f;
    for (uint32_t e = 0; e < members; e++) {
      const float v = y[((uint64_t)e * rows + row) * cols + c] * s + b;
      a = e == 0 ? v : a + v;
      a2 = e == 0 ? v * v : a2 + v * v;
    }
    const float m = a * inv_e;
    const float d = sqrtf(fmaxf(a2 * inv_e - m * m, 0.0f));
    const uint64_t i = (uint64_t)row * cols + c;
    out_mean[i] = m;
    if (out_std) out_std[i] = d;
    if (m >= level) most = fmaxf(most, d);
  }
  for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  if (lane == 0 && out_spread) out_spread[row] = most;
}

}  // namespace

// A launch whose blocks may start before the stream's last kernel has ended (they
// call tc::grid_wait): the three launches of a training step then follow each
// other without the gaps of 3 to 4 us (132 -> 125 us a step, with the optimizer's
// quads a thread each and one image store a quad; 10,000 rows of inference 222 ->
// 213 us, a gradient of 4096 rows 188 -> 181 us).
template <class... P, class... A>
static cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, uint32_t threads, uint32_t smem, cudaStream_t s,
                                  A&&... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

// The kernels' shared-memory limits (call it outside any stream capture,
// before the first launch on a device; repeating it is harmless).
cudaError_t mlp_net_init() {
  cudaError_t e = cudaFuncSetAttribute(rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem<false>);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem<true>);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwSmem);
}

cudaError_t launch_mlp_rows(const MlpRowsArgs& a, uint32_t members, bool train, cudaStream_t s) {
  if (a.rows == 0 || members == 0) return cudaSuccess;
  const dim3 grid((a.rows + kRows - 1) / kRows, members);
  return launch_chained(train ? rows_kernel<true> : rows_kernel<false>, grid, kRowThreads,
                        train ? kRowsSmem<true> : kRowsSmem<false>, s, a);
}

// The shares of a batch's rows that a weight gradient is summed in: 512 rows each up
// to eight of them, then an eighth, in multiples of 64. A sum's partition is part of
// its result: AdamW makes whole steps of the roundings of near-zero gradients, so it
// depends on the batch alone, not on the members or the chip.
uint32_t dw_shares(uint32_t rows, uint32_t& share_rows) {
  const uint32_t n = std::max(1u, std::min(8u, rows / 512u));
  share_rows = ((rows + n - 1u) / n + 63u) / 64u * 64u;
  return (rows + share_rows - 1u) / share_rows;
}

cudaError_t launch_mlp_dw(MlpDwArgs a, int n_sms, cudaStream_t s) {
  const uint32_t L = a.net.n_layers;
  uint32_t wide = 0, first = 0, width = 0;     // (member, feature block, input block) units; the widest input block
  for (uint32_t l = 0; l < L; l++) {
    const MlpLayerDesc& D = a.net.L[l];
    const uint32_t units = ((D.op + 127u) / 128u) * ((D.ip + kWide - 1) / kWide) * a.members;
    (l == 0 ? first : wide) += units;
    if (l > 0) width = std::max(width, D.ip);
  }
  const uint32_t width0 = std::min(kWide, a.net.L[0].ip);
  a.shares = dw_shares(a.tiles * kRows, a.share_rows);
  // Shares a CTA, for the layers beyond the first and for the first, narrower one: as
  // many as TMEM holds at most, and those whose largest CTA loads the least with all
  // CTAs on the chip at once; where that cannot be, by the bound of a list schedule.
  const uint32_t most = std::min(a.shares, kDwTmem / dw_columns(width)),
                 most0 = std::min(a.shares, kDwTmem / dw_columns(width0));
  uint64_t best = ~0ull;
  for (uint32_t g = 1; g <= most; g++)
    for (uint32_t g0 = 1; g0 <= most0; g0++) {
      const uint64_t c = (uint64_t)g * (128u + width), c0 = (uint64_t)g0 * (128u + width0);
      const uint64_t n = (uint64_t)wide * ((a.shares + g - 1) / g), n0 = (uint64_t)first * ((a.shares + g0 - 1) / g0);
      uint64_t cost = std::max(c, c0);
      if (n + n0 > (uint64_t)n_sms) cost += (n * c + n0 * c0) / (uint64_t)n_sms;
      if (cost < best) {
        best = cost;
        a.group = g;
        a.group0 = g0;
      }
    }
  const uint32_t blocks = wide * ((a.shares + a.group - 1) / a.group) + first * ((a.shares + a.group0 - 1) / a.group0);
  return launch_chained(dw_kernel, dim3(blocks), kDwThreads, kDwSmem, s, a);
}

cudaError_t launch_mlp_adamw(const MlpAdamwArgs& a, cudaStream_t s) {
  return launch_chained(adamw_kernel, dim3((a.net.p_stride / 4u + 255u) / 256u, a.net.members), 256, 0, s, a);
}

cudaError_t launch_mlp_images(const MlpNet& net, const float* P, uint16_t* img, cudaStream_t s) {
  const dim3 grid(std::min(1024u, (net.p_stride + 255u) / 256u), net.members);
  image_kernel<<<grid, 256, 0, s>>>(net, P, img);
  return cudaGetLastError();
}

cudaError_t launch_mlp_ensemble(const float* y, uint32_t members, uint32_t rows, uint32_t cols, const float* mean,
                                const float* sd, float level, float* out_mean, float* out_std, float* out_spread,
                                cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  return launch_chained(ensemble_kernel, dim3((rows + 7) / 8), 256, 0, s, y, members, rows, cols, mean, sd,
                        1.0f / (float)members, level, out_mean, out_std, out_spread);
}

}  // namespace omg
