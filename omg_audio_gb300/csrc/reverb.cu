// estimate_reverb on the GPU (crates/omg-core/src/tracer.rs:204-257): one
// block per (echogram, band). FP64 is used only here, for the Schroeder
// backward integral and the line fit. The late level is the reference's own
// f32 sum of the bins from 80 ms on, in its order (tracer.rs:246-254).
//
// What bounds it: serial chains. The FP64 unit takes a warp's add 16 cycles
// and returns it some 40 later, so one warp per band (chunks of 63 bins of a
// 2000-bin curve summed one after another, twice) took 49 us for one job and
// 108 us for 64. Here four warps sum chunks a quarter as long, a
// block-wide scan joins them, and one further warp runs the late level's
// sequential f32 sum (4 cycles an add, its loads ahead of it) beside them.
// Shared memory holds one 8-byte slot a bin: the bin, then its place on the
// curve. Once there are more curves than multiprocessors the chip has other blocks to
// run, and four warps' scans and logarithms are four times one's (reverb_few).
#include <cfloat>

#include "omg_internal.h"

namespace omg {

namespace {

__device__ __forceinline__ double db_of(double e, double total) {
  return 10.0 * log10(fmax(e / total, 1e-12));
}

// the W warps of the decay curve only (named barrier 1)
template <uint32_t W>
__device__ __forceinline__ void edc_sync() {
  if (W == 1) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"n"(32u * W) : "memory");
}

// W: warps of the decay curve; the last warp is the late level's.
template <uint32_t W>
__global__ void __launch_bounds__(32 * W + 32)
    reverb_kernel(const DReverbJob* __restrict__ rj, uint32_t n_jobs, const float* __restrict__ bins,
                  omg_reverb* __restrict__ out, const uint32_t* __restrict__ job_segments) {
  extern __shared__ double edc[];           // n bins: first as f32 in each slot's low word, then the FP64 curve
  __shared__ double s_tot[W];
  __shared__ uint32_t s_f5[W], s_f25[W], s_neg[W];
  __shared__ double s_fit[4][W];
  const uint32_t j = blockIdx.x, b = blockIdx.y;
  const DReverbJob R = rj[j];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (j >= n_jobs) return;
  if (b >= R.nb) {
    if (b < OMG_MAX_BANDS && tid == 0) {
      out[j].rt60[b] = 0.0f;
      out[j].level[b] = 0.0f;
      out[j].rt60_fit[b] = 0.0f;
    }
    return;
  }
  const uint32_t n = R.n_bins, nb = R.nb;
  const float* B = bins + R.bins_off;

  if (warp == W) {
    // tracer.rs:246: late_start = (0.080 / BIN_DT) as usize in f32. The warp
    // loads kAhead groups of 32 bins while it adds the previous ones, bin after
    // bin, every lane the same sum.
    constexpr uint32_t kAhead = 4;
    const float q = 0.080f / R.bin_dt;
    const uint64_t ls = (q >= 0.0f) ? (uint64_t)q : 0;
    float late = 0.0f;
    if (ls < n) {
      float cur[kAhead], nxt[kAhead];
      auto load = [&](float (&v)[kAhead], uint32_t i0) {
#pragma unroll
        for (uint32_t g = 0; g < kAhead; g++) {
          const uint32_t i = i0 + 32u * g + lane;
          v[g] = i < n ? B[(uint64_t)i * nb + b] : 0.0f;
        }
      };
      load(cur, (uint32_t)ls);
      for (uint32_t i0 = (uint32_t)ls; i0 < n; i0 += 32u * kAhead) {
        load(nxt, i0 + 32u * kAhead);
#pragma unroll
        for (uint32_t g = 0; g < kAhead; g++) {
          const uint32_t left = n - min(n, i0 + 32u * g);
          if (left >= 32u) {
#pragma unroll
            for (int k = 0; k < 32; k++) late += __shfl_sync(0xffffffffu, cur[g], k);
          } else {
            for (uint32_t k = 0; k < left; k++) late += __shfl_sync(0xffffffffu, cur[g], (int)k);
          }
          cur[g] = nxt[g];
        }
      }
    }
    if (lane == 0) {
      out[j].level[b] = fminf(sqrtf(late), 0.7f);
      if (b == 0) out[j].segments = job_segments ? job_segments[rj[j].seg] : 0;
    }
    return;
  }

  bool neg = false;
  for (uint32_t i = tid; i < n; i += 32u * W) {
    const float v = B[(uint64_t)i * nb + b];
    neg |= v < 0.0f;
    reinterpret_cast<float*>(edc)[2u * i] = v;
  }
  neg = __any_sync(0xffffffffu, neg);
  if (lane == 0) s_neg[warp] = neg ? 1u : 0u;
  edc_sync<W>();
  bool any_neg = false;
  for (uint32_t w = 0; w < W; w++) any_neg |= s_neg[w] != 0u;

  // per-thread contiguous chunk, sequential backward sum, then an exclusive
  // suffix scan of the chunk totals over the block
  const uint32_t chunk = (n + 32u * W - 1u) / (32u * W);
  const uint32_t lo = min(n, tid * chunk), hi = min(n, lo + chunk);
  double run = 0.0;
  for (int64_t i = (int64_t)hi - 1; i >= (int64_t)lo; i--) {
    run += (double)reinterpret_cast<const float*>(edc)[2 * i];
    edc[i] = run;
  }
  double incl = run;
  for (int off = 1; off < 32; off <<= 1) {
    const double v = __shfl_down_sync(0xffffffffu, incl, off);
    if (lane + off < 32) incl += v;
  }
  if (lane == 0) s_tot[warp] = incl;
  double after = __shfl_down_sync(0xffffffffu, incl, 1);
  if (lane == 31) after = 0.0;
  edc_sync<W>();
  double later = 0.0;
  for (uint32_t w = W - 1; w > warp; w--) later += s_tot[w];
  after += later;
  for (uint32_t i = lo; i < hi; i++) edc[i] += after;
  edc_sync<W>();
  const double total = edc[0];

  float rt60 = 0.5f, fit = 0.5f;
  if (total > 0.0) {
    // first bins at <= -5 dB and <= -25 dB. The curve of bins that are not
    // negative does not rise, so a chunk whose last bin is above -5 dB holds
    // neither. The dB value is computed only for a bin within 1e-9 (relative)
    // of a level's energy: elsewhere the energy ratio decides the same
    // comparison, without a logarithm per bin.
    const double r5 = sqrt(0.1);            // 10^(-5/10)
    const double e5 = total * r5, e25 = total * (r5 * 0.01);
    auto below = [&](double e, double level, double thr) {
      if (e < thr * (1.0 - 1e-9)) return true;
      if (e > thr * (1.0 + 1e-9)) return false;
      return db_of(e, total) <= level;
    };
    uint32_t f5 = 0xFFFFFFFFu, f25 = 0xFFFFFFFFu;
    if (lo < hi && (any_neg || below(edc[hi - 1], -5.0, e5))) {
      for (uint32_t i = lo; i < hi && f25 == 0xFFFFFFFFu; i++) {
        const double e = edc[i];
        if (f5 == 0xFFFFFFFFu && below(e, -5.0, e5)) f5 = i;
        if (below(e, -25.0, e25)) f25 = i;
      }
    }
    f5 = __reduce_min_sync(0xffffffffu, f5);
    f25 = __reduce_min_sync(0xffffffffu, f25);
    if (lane == 0) {
      s_f5[warp] = f5;
      s_f25[warp] = f25;
    }
    edc_sync<W>();
    for (uint32_t w = 0; w < W; w++) {
      f5 = min(f5, s_f5[w]);
      f25 = min(f25, s_f25[w]);
    }
    // the reference stops scanning at t25, so t5 is only set when found first
    if (f25 != 0xFFFFFFFFu && f5 != 0xFFFFFFFFu && f5 <= f25 && f25 > f5) {
      const double d5 = db_of(edc[f5], total), d25 = db_of(edc[f25], total);
      const float dt = (float)(f25 - f5) * R.bin_dt;
      const float ddb = (float)(d25 - d5);
      rt60 = fminf(fmaxf(-60.0f * dt / ddb, 0.1f), 5.0f);
      // least-squares T20 line of dB(EDC) over [t5, t25]
      double sx = 0, sy = 0, sxx = 0, sxy = 0;
      for (uint32_t i = f5 + tid; i <= f25; i += 32u * W) {
        const double x = (double)i * (double)R.bin_dt, y = db_of(edc[i], total);
        sx += x; sy += y; sxx += x * x; sxy += x * y;
      }
      for (int off = 16; off > 0; off >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, off);
        sy += __shfl_xor_sync(0xffffffffu, sy, off);
        sxx += __shfl_xor_sync(0xffffffffu, sxx, off);
        sxy += __shfl_xor_sync(0xffffffffu, sxy, off);
      }
      if (lane == 0) {
        s_fit[0][warp] = sx;
        s_fit[1][warp] = sy;
        s_fit[2][warp] = sxx;
        s_fit[3][warp] = sxy;
      }
      edc_sync<W>();
      if (tid == 0) {
        sx = sy = sxx = sxy = 0.0;
        for (uint32_t w = 0; w < W; w++) {
          sx += s_fit[0][w];
          sy += s_fit[1][w];
          sxx += s_fit[2][w];
          sxy += s_fit[3][w];
        }
        const double cnt = (double)(f25 - f5 + 1);
        const double den = cnt * sxx - sx * sx;
        if (den > 0) {
          const double slope = (cnt * sxy - sx * sy) / den;
          if (slope < 0) fit = (float)fmin(fmax(-60.0 / slope, 0.1), 5.0);
        }
      }
    }
  }
  if (tid == 0) {
    out[j].rt60[b] = rt60;
    out[j].rt60_fit[b] = fit;
  }
}

// Whether four warps take a curve, or one. A call of three bands a job, us (one warp,
// then four): 64 jobs of 300 bins 53, 54, of 2000 bins 123, 99; 128 of 300 bins 55, 68, of
// 1000 bins 98, 98; 512 of 2000 bins 346, 354, of 8000 bins 1480, 1200; 4096 of 300 bins
// 482, 754. Beyond 4096 bins a curve's shared memory holds few blocks a multiprocessor
// whatever their warps.
bool reverb_few(uint32_t n_jobs, uint32_t nb, uint32_t max_bins) {
  const uint64_t curves = (uint64_t)n_jobs * nb;
  return curves <= 152u || max_bins > 4096u || (curves <= 384u && max_bins >= 768u);
}

}  // namespace

cudaError_t launch_reverb(const DReverbJob* rj, uint32_t n_jobs, uint32_t nb, uint32_t max_bins, const float* bins,
                          omg_reverb* out, const uint32_t* job_segments, cudaStream_t s) {
  if (n_jobs == 0) return cudaSuccess;
  if (max_bins > kMaxBins) return cudaErrorInvalidValue;
  const size_t smem = (size_t)max_bins * sizeof(double);
  const bool few = reverb_few(n_jobs, nb, max_bins);
  if (smem > 40 * 1024) {   // beyond the default limit with the block's own few arrays
    cudaError_t e = cudaFuncSetAttribute(few ? reverb_kernel<4> : reverb_kernel<1>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid(n_jobs, OMG_MAX_BANDS);
  if (few)
    reverb_kernel<4><<<grid, 32 * 4 + 32, smem, s>>>(rj, n_jobs, bins, out, job_segments);
  else
    reverb_kernel<1><<<grid, 32 + 32, smem, s>>>(rj, n_jobs, bins, out, job_segments);
  return cudaGetLastError();
}

}  // namespace omg
