// C ABI of the GB300 tracer (include/omg_cuda.h), part 4: the learned
// surrogate. An ensemble of MLPs (n_in -> hidden x n_hidden -> n_out, GELU)
// trained and run by the tensor-core kernels of mlp_net.cu: BF16 weights and
// activations, FP32 accumulation, FP32 master weights, AdamW with a cosine
// learning-rate decay, MSE on standardized targets. Inference returns the
// ensemble mean and spread in the caller's units.
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>

#include "mlp_net.h"
#include "runtime.h"

using namespace omg;

namespace omg {

// Scratch of one launch of `tiles` 128-row tiles of `members` members
// (MlpRowsArgs): the images that the weight gradients read, GELU'(Z), the bias
// gradients' sums of 32 rows.
struct MlpScratch {
  uint64_t tiles = 0;              // members x tiles
  DevBuf<uint16_t> xt, at, dzt;
  DevBuf<float> gz, gb;
};

// One of the two chunks of rows in flight during inference.
struct MlpChunk {
  DevBuf<float> y, mean, std, spread;      // y: [member][row][out]; each grown by its own size (std by predict alone)
  cudaEvent_t done = nullptr;
  ~MlpChunk() {
    if (done) cudaEventDestroy(done);
  }
};

struct MlpRec {
  omg_mlp_config cfg{};
  MlpNet net{};
  // every member's parameters, AdamW moments and gradients (net.p_stride floats a member), the
  // weights' bf16 images
  DevBuf<float> P, M1, V1, G;
  DevBuf<uint16_t> img;
  DevBuf<float> loss;                           // per member
  // standardization (host and device)
  std::vector<float> x_mean, x_std, y_mean, y_std;
  DevBuf<float> d_x_mean, d_x_std, d_y_mean, d_y_std;
  // inference: a group's inputs, two chunks' outputs, the stream of the copies back
  DevBuf<float> xin;
  MlpChunk chunk[2];
  PinBuf<float> h_small;                        // a small call's results (kSmallFloats)
  cudaStream_t back = nullptr;
  MlpScratch train_s, grad_s;
  DevBuf<float> grad_x, grad_y;                 // omg_mlp_grad's batch
  // dataset (standardized, device)
  uint32_t n_data = 0;
  DevBuf<float> X, Y;
  uint64_t step = 0;
  DevBuf<float> sched;                          // per step: learning rate, bias corrections 1 and 2
  DevBuf<uint32_t> perm, counters;              // two epochs' permutations; step counter, ticket
  PinBuf<uint32_t> h_perm;
  DevBuf<float> epoch_loss;
  DevBuf<uint32_t> err;
  PinBuf<uint32_t> h_err;
  ~MlpRec() {
    if (back) cudaStreamDestroy(back);
  }
  PinBuf<float> h_loss;
};

}  // namespace omg

namespace {

// Results of at most this many floats come back through pinned memory, behind the
// kernels: two copies into pageable memory, one after the other behind a wait, took 6
// to 14 us more (a row of 1-16x1-1 57 us against 40, of 1024-64x2-8 104 against 81).
constexpr uint64_t kSmallFloats = 1u << 14;

constexpr uint32_t kGraphSteps = 8;   // training steps recorded in one graph

uint32_t n_layers(const MlpRec& M) { return M.cfg.n_hidden + 1; }

// The layout of one member (MlpLayerDesc).
MlpNet make_net(const omg_mlp_config& c) {
  MlpNet N{};
  N.n_layers = c.n_hidden + 1;
  N.members = c.members;
  uint32_t in = c.n_in, p = 0, im = 0;
  for (uint32_t l = 0; l < N.n_layers; l++) {
    MlpLayerDesc& D = N.L[l];
    D.in = in;
    D.out = l + 1 == N.n_layers ? c.n_out : c.hidden;
    D.ip = (D.in + 15u) & ~15u;
    D.op = (D.out + 15u) & ~15u;
    D.w_off = p;
    p += (D.in * D.out + 3u) & ~3u;
    D.b_off = p;
    p += (D.out + 3u) & ~3u;
    D.img_off = im;
    im += D.ip * D.op;
    in = D.out;
  }
  N.p_stride = p;
  N.img_stride = im;
  return N;
}

int32_t ensure_scratch(omg_ctx* ctx, const MlpRec& M, MlpScratch& S, uint64_t tiles) {
  if (tiles <= S.tiles) return OMG_OK;
  const uint32_t L = n_layers(M);
  S.tiles = 0;
  CK(S.xt.alloc(tiles * 128u * M.net.L[0].ip));
  CK(S.at.alloc(tiles * (L - 1) * 128u * M.cfg.hidden));
  CK(S.dzt.alloc(tiles * L * 128u * kMlpWide));
  CK(S.gz.alloc(tiles * (L - 1) * 128u * M.cfg.hidden));
  CK(S.gb.alloc(tiles * 4u * L * kMlpWide));
  S.tiles = tiles;
  return OMG_OK;
}

// The launch arguments of a training pass of `rows` rows from X, Y (standardized) through scratch S.
MlpRowsArgs rows_args(const MlpRec& M, const MlpScratch& S, const float* X, const float* Y, uint32_t rows,
                      uint32_t member0) {
  MlpRowsArgs a{};
  a.net = M.net;
  a.rows = rows;
  a.member0 = member0;
  a.P = M.P.p;
  a.img = M.img.p;
  a.X = X;
  a.Y = Y;
  a.loss = M.loss.p;
  a.xt = S.xt.p;
  a.at = S.at.p;
  a.dzt = S.dzt.p;
  a.gz = S.gz.p;
  a.gb = S.gb.p;
  a.err = M.err.p;
  return a;
}

MlpDwArgs dw_args(const MlpRec& M, const MlpScratch& S, uint32_t rows, uint32_t members, uint32_t member0) {
  MlpDwArgs a{};
  a.net = M.net;
  a.tiles = rows / 128u;
  a.members = members;
  a.member0 = member0;
  a.G = M.G.p;
  a.xt = S.xt.p;
  a.at = S.at.p;
  a.dzt = S.dzt.p;
  a.gb = S.gb.p;
  a.err = M.err.p;
  return a;
}

// The kernels' error word, brought to M.h_err behind the work on stream s; then, once that is done, its meaning.
cudaError_t fetch_err(MlpRec& M, cudaStream_t s) {
  return cudaMemcpyAsync(M.h_err.p, M.err.p, 4, cudaMemcpyDeviceToHost, s);
}
int32_t check_err(omg_ctx* ctx, MlpRec& M) {
  if (*M.h_err.p) {
    ctx->last_error = "surrogate network: an mbarrier wait ran out";
    CK(cudaMemsetAsync(M.err.p, 0, 4, ctx->stream));
    return OMG_E_TIMEOUT;
  }
  return OMG_OK;
}

int32_t sync_norm(omg_ctx* ctx, MlpRec& M) {
  if (!M.d_x_mean.p) {
    CK(M.d_x_mean.alloc(M.cfg.n_in));
    CK(M.d_x_std.alloc(M.cfg.n_in));
    CK(M.d_y_mean.alloc(M.cfg.n_out));
    CK(M.d_y_std.alloc(M.cfg.n_out));
  }
  CK(cudaMemcpy(M.d_x_mean.p, M.x_mean.data(), M.cfg.n_in * 4, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(M.d_x_std.p, M.x_std.data(), M.cfg.n_in * 4, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(M.d_y_mean.p, M.y_mean.data(), M.cfg.n_out * 4, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(M.d_y_std.p, M.y_std.data(), M.cfg.n_out * 4, cudaMemcpyHostToDevice));
  return OMG_OK;
}

// Copy between packed host arrays and a member's padded block: W then b per layer.
template <class F>
void each_param(const MlpNet& N, F&& f) {
  for (uint32_t l = 0; l < N.n_layers; l++) {
    f(N.L[l].w_off, N.L[l].in * N.L[l].out);
    f(N.L[l].b_off, N.L[l].out);
  }
}

bool valid_cfg(const omg_mlp_config& c) {
  return c.n_in >= 1 && c.n_in <= 1024 && c.hidden >= 16 && c.hidden <= 256 && c.hidden % 16 == 0 &&
         c.n_hidden >= 1 && c.n_hidden <= 16 && c.n_out >= 1 && c.n_out <= 256 && c.members >= 1 &&
         c.members <= 16;
}

}  // namespace

extern "C" {

int32_t omg_mlp_create(omg_ctx* ctx, const omg_mlp_config* cfg, uint32_t* id) {
  if (!ctx || !cfg || !id || !valid_cfg(*cfg)) return OMG_E_INVALID;
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(ctx, cudaGetLastError(), "cudaSetDevice");
  CK(mlp_net_init());
  std::shared_ptr<MlpRec> M(new MlpRec());
  M->cfg = *cfg;
  M->net = make_net(*cfg);
  const MlpNet& N = M->net;
  const uint32_t L = N.n_layers;
  std::mt19937_64 rng(cfg->seed ? cfg->seed : 1u);
  const size_t np = (size_t)N.p_stride * cfg->members, ni = (size_t)N.img_stride * cfg->members;
  std::vector<float> p0(np, 0.0f);
  for (uint32_t e = 0; e < cfg->members; e++) {
    for (uint32_t l = 0; l < L; l++) {
      const MlpLayerDesc& D = N.L[l];
      // He-style normal init (std sqrt(2 / fan_in)), zero biases
      std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)D.in));
      float* w = p0.data() + (size_t)e * N.p_stride + D.w_off;
      const size_t nw = (size_t)D.out * D.in;
      for (size_t i = 0; i < nw; i++) w[i] = nd(rng);
      if (l + 1 == L)
        for (size_t i = 0; i < nw; i++) w[i] *= 0.5f;
    }
  }
  CK(M->P.alloc(np));
  CK(M->M1.alloc(np));
  CK(M->V1.alloc(np));
  CK(M->G.alloc(np));
  CK(M->img.alloc(ni));
  CK(M->loss.alloc(cfg->members));
  CK(cudaMemcpy(M->P.p, p0.data(), np * 4, cudaMemcpyHostToDevice));
  CK(cudaMemsetAsync(M->M1.p, 0, np * 4, ctx->stream));
  CK(cudaMemsetAsync(M->V1.p, 0, np * 4, ctx->stream));
  CK(cudaMemsetAsync(M->G.p, 0, np * 4, ctx->stream));
  CK(cudaMemsetAsync(M->img.p, 0, ni * 2, ctx->stream));   // the images' padding stays zero
  CK(launch_mlp_images(N, M->P.p, M->img.p, ctx->stream));
  M->x_mean.assign(cfg->n_in, 0.0f);
  M->x_std.assign(cfg->n_in, 1.0f);
  M->y_mean.assign(cfg->n_out, 0.0f);
  M->y_std.assign(cfg->n_out, 1.0f);
  CK(M->err.alloc(1));
  CK(M->h_err.alloc(1));
  CK(M->h_loss.alloc(1));
  CK(cudaMemsetAsync(M->err.p, 0, 4, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  int32_t rc = sync_norm(ctx, *M);
  if (rc) return rc;
  *id = ctx->next_mlp++;
  ctx->mlps[*id] = M;
  return OMG_OK;
}

int32_t omg_mlp_destroy(omg_ctx* ctx, uint32_t id) {
  if (!ctx) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  cudaStreamSynchronize(ctx->stream);
  ctx->mlps.erase(it);
  return OMG_OK;
}

int32_t omg_mlp_set_data(omg_ctx* ctx, uint32_t id, const float* x, const float* y, uint32_t n) {
  if (!ctx || !x || !y || n == 0) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  const uint32_t ni = M.cfg.n_in, no = M.cfg.n_out;
  // standardization from the data (FP64 sums)
  for (int which = 0; which < 2; which++) {
    const float* d = which ? y : x;
    const uint32_t c = which ? no : ni;
    std::vector<double> s(c, 0.0), q(c, 0.0);
    for (uint64_t i = 0; i < n; i++)
      for (uint32_t k = 0; k < c; k++) {
        const double v = d[i * c + k];
        if (!std::isfinite(v)) return OMG_E_INVALID;
        s[k] += v;
        q[k] += v * v;
      }
    std::vector<float>& mean = which ? M.y_mean : M.x_mean;
    std::vector<float>& sd = which ? M.y_std : M.x_std;
    for (uint32_t k = 0; k < c; k++) {
      const double m = s[k] / n, var = std::max(q[k] / n - m * m, 0.0);
      mean[k] = (float)m;
      sd[k] = (float)std::max(std::sqrt(var), 1e-6);
    }
  }
  std::vector<float> xs((size_t)n * ni), ys((size_t)n * no);
  for (uint64_t i = 0; i < n; i++) {
    for (uint32_t k = 0; k < ni; k++) xs[i * ni + k] = (x[i * ni + k] - M.x_mean[k]) / M.x_std[k];
    for (uint32_t k = 0; k < no; k++) ys[i * no + k] = (y[i * no + k] - M.y_mean[k]) / M.y_std[k];
  }
  int32_t rc = sync_norm(ctx, M);
  if (rc) return rc;
  M.n_data = 0;   // (until both are there)
  CK(M.X.alloc(xs.size()));
  CK(M.Y.alloc(ys.size()));
  CK(cudaMemcpy(M.X.p, xs.data(), xs.size() * 4, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(M.Y.p, ys.data(), ys.size() * 4, cudaMemcpyHostToDevice));
  M.n_data = n;
  return OMG_OK;
}

// Training: three launches a step for all members together (the rows' forward
// and backward pass, the weight gradients, AdamW), recorded into a CUDA graph
// that is launched steps-per-epoch times per epoch. The step's batch rows (the
// epoch's permutation) and its learning rate and bias corrections (a schedule
// uploaded once) are read on the device at the step counter. Two epochs'
// permutations are resident: the host shuffles the next epoch's, a thread a
// member, while the device runs this one.
int32_t omg_mlp_train(omg_ctx* ctx, uint32_t id, const omg_mlp_train_config* tc, float* epoch_loss) {
  if (!ctx || !tc || tc->epochs == 0 || tc->batch == 0 || tc->batch % 128 != 0) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  if (M.n_data < tc->batch) return OMG_E_INVALID;
  const uint32_t B = tc->batch, E = M.cfg.members, n = M.n_data;
  const uint32_t spe = n / B;
  const uint64_t total = (uint64_t)spe * tc->epochs;
  if (total >= (1ull << 31)) return OMG_E_INVALID;
  // the schedule: cosine decay from lr to lr_final, AdamW bias corrections
  std::vector<float> sched(3 * total);
  for (uint64_t t = 0; t < total; t++) {
    const double prog = total > 1 ? (double)t / (double)(total - 1) : 1.0;
    sched[3 * t] = (float)(tc->lr_final + 0.5 * (tc->lr - tc->lr_final) * (1.0 + std::cos(3.14159265358979323846 * prog)));
    sched[3 * t + 1] = (float)(1.0 - std::pow((double)tc->beta1, (double)(t + 1)));
    sched[3 * t + 2] = (float)(1.0 - std::pow((double)tc->beta2, (double)(t + 1)));
  }
  CK(mlp_net_init());   // outside the capture below
  cudaStream_t s = ctx->stream;
  const uint64_t half = (uint64_t)E * n, n_loss = (uint64_t)E * tc->epochs;
  CK(cudaStreamSynchronize(s));
  if (M.sched.n < sched.size()) CK(M.sched.alloc(sched.size()));
  if (M.perm.n < 2 * half) CK(M.perm.alloc(2 * half));
  if (M.h_perm.n < 2 * half) CK(M.h_perm.alloc(2 * half));
  if (!M.counters.p) CK(M.counters.alloc(2));
  if (M.epoch_loss.n < n_loss) CK(M.epoch_loss.alloc(n_loss));
  int32_t rc = ensure_scratch(ctx, M, M.train_s, (uint64_t)E * (B / 128u));
  if (rc) return rc;
  CK(cudaMemcpyAsync(M.sched.p, sched.data(), sched.size() * 4, cudaMemcpyHostToDevice, s));
  CK(cudaMemsetAsync(M.counters.p, 0, 8, s));
  CK(cudaMemsetAsync(M.G.p, 0, M.G.n * 4, s));          // each step leaves them zero again
  CK(cudaMemsetAsync(M.loss.p, 0, M.loss.n * 4, s));
  MlpRowsArgs ra = rows_args(M, M.train_s, M.X.p, M.Y.p, B, 0);
  ra.perm = M.perm.p;
  ra.perm_half = half;
  ra.perm_member = n;
  ra.step = M.counters.p;
  ra.spe = spe;
  MlpAdamwArgs aa{};
  aa.net = M.net;
  aa.P = M.P.p;
  aa.M1 = M.M1.p;
  aa.V1 = M.V1.p;
  aa.G = M.G.p;
  aa.img = M.img.p;
  aa.sched = M.sched.p;
  aa.step = M.counters.p;
  aa.ticket = M.counters.p + 1;
  aa.loss = M.loss.p;
  aa.epoch_loss = M.epoch_loss.p;
  aa.spe = spe;
  aa.epochs = tc->epochs;
  aa.b1 = tc->beta1;
  aa.b2 = tc->beta2;
  aa.eps = tc->eps;
  aa.wd = tc->weight_decay;
  // two graphs: kGraphSteps steps (the gap between two graphs is some us), and one step for the rest of an epoch
  const uint32_t per_graph[2] = {std::min(spe, kGraphSteps), 1u};
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  {
    cudaStream_t cs;
    CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t ce = cudaSuccess;
    for (int k = 0; k < 2 && ce == cudaSuccess; k++) {
      if (k == 1 && spe % per_graph[0] == 0) break;
      ce = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
      if (ce != cudaSuccess) break;
      for (uint32_t i = 0; i < per_graph[k] && ce == cudaSuccess; i++) {
        ce = launch_mlp_rows(ra, E, true, cs);
        if (ce == cudaSuccess) ce = launch_mlp_dw(dw_args(M, M.train_s, B, E, 0), ctx->n_sms, cs);
        if (ce == cudaSuccess) ce = launch_mlp_adamw(aa, cs);
      }
      cudaGraph_t g = nullptr;
      const cudaError_t ee = cudaStreamEndCapture(cs, &g);
      if (ce == cudaSuccess) ce = ee;
      if (ce == cudaSuccess) ce = cudaGraphInstantiate(&graph[k], g, 0);
      if (g) cudaGraphDestroy(g);
    }
    cudaStreamDestroy(cs);
    if (ce != cudaSuccess) {
      for (cudaGraphExec_t g : graph)
        if (g) cudaGraphExecDestroy(g);
      return fail(ctx, ce, "training step capture");
    }
  }
  std::vector<std::mt19937_64> rngs;
  for (uint32_t e = 0; e < E; e++) rngs.emplace_back((tc->seed ? tc->seed : 7u) + 0x9E3779B97F4A7C15ull * e);
  auto shuffle_epoch = [&](uint32_t ep) {
    const int threads = (uint64_t)E * n >= 4096u ? (int)E : 1;
#pragma omp parallel for num_threads(threads) schedule(static)
    for (int e = 0; e < (int)E; e++) {
      uint32_t* p = M.h_perm.p + (ep & 1u) * half + (uint64_t)e * n;
      std::iota(p, p + n, 0u);
      std::shuffle(p, p + n, rngs[e]);
    }
  };
  // from here on every exit waits for what was enqueued: it reads sched and the permutations
  cudaError_t ce = cudaSuccess;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  for (int k = 0; k < 2 && ce == cudaSuccess; k++) ce = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
  for (uint32_t ep = 0; ep < tc->epochs && ce == cudaSuccess; ep++) {
    // this half's previous epoch (two before) is done with its permutations
    if (ep >= 2) ce = cudaEventSynchronize(ev[ep & 1u]);
    if (ce != cudaSuccess) break;
    shuffle_epoch(ep);
    const uint64_t at = (ep & 1u) * half;
    ce = cudaMemcpyAsync(M.perm.p + at, M.h_perm.p + at, half * 4, cudaMemcpyHostToDevice, s);
    for (uint32_t st = 0; st < spe && ce == cudaSuccess;) {
      const int k = spe - st >= per_graph[0] ? 0 : 1;
      ce = cudaGraphLaunch(graph[k], s);
      st += per_graph[k];
    }
    if (ce == cudaSuccess) ce = cudaEventRecord(ev[ep & 1u], s);
  }
  std::vector<float> losses(n_loss);
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(losses.data(), M.epoch_loss.p, n_loss * 4, cudaMemcpyDeviceToHost, s);
  if (ce == cudaSuccess) ce = fetch_err(M, s);
  const cudaError_t se = cudaStreamSynchronize(s);
  for (int k = 0; k < 2; k++)
    if (ev[k]) cudaEventDestroy(ev[k]);
  for (cudaGraphExec_t g : graph)
    if (g) cudaGraphExecDestroy(g);
  if (ce != cudaSuccess) return fail(ctx, ce, "training");
  if (se != cudaSuccess) return fail(ctx, se, "training");
  if (epoch_loss) std::copy(losses.begin(), losses.end(), epoch_loss);
  M.step += total;
  return check_err(ctx, M);
}

}  // extern "C"

namespace {

// Shared by omg_surrogate_predict and omg_surrogate_query: y_std (full
// spread) and/or row_spread (per row, the largest spread among outputs whose
// mean is >= level) are optional.
int32_t surrogate_run(omg_ctx* ctx, uint32_t id, const float* x, uint32_t n, float* y_mean, float* y_std,
                      float* row_spread, float level) {
  if (!ctx || !x || !y_mean || n == 0) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  const uint32_t ni = M.cfg.n_in, no = M.cfg.n_out, E = M.cfg.members;
  // Rows a launch (chunk): the row tiles of all members fill the chip once (one
  // CTA a multiprocessor). Two chunks are in flight: one's results are copied
  // straight into the caller's arrays while the other's kernels run (8 MB from
  // the device into pageable memory take 60 us on the GB300's host, a copy
  // through pinned memory 53 us and 170 us more for the host's part). The
  // inputs go up for up to kGroup chunks at a time.
  constexpr uint32_t kGroup = 8;
  const uint32_t wave = 128u * std::max(1u, (uint32_t)ctx->n_sms / E);
  const uint32_t parts = (n + wave - 1) / wave;
  const uint32_t chunk = std::min(n, ((n + parts - 1) / parts + 127u) / 128u * 128u);
  const uint64_t group = (uint64_t)chunk * kGroup, n_mean = (uint64_t)n * no, n_std = y_std ? n_mean : 0,
                 n_spread = row_spread ? n : 0;
  const bool small = n <= chunk && n_mean + n_std + n_spread <= kSmallFloats;
  cudaStream_t s = ctx->stream;
  if (small && !M.h_small.p) CK(M.h_small.alloc(kSmallFloats));
  if (!M.back) CK(cudaStreamCreateWithFlags(&M.back, cudaStreamNonBlocking));
  if (M.xin.n < std::min<uint64_t>(n, group) * ni) CK(M.xin.alloc(std::min<uint64_t>(n, group) * ni));
  for (int k = 0; k < (n > chunk ? 2 : 1); k++) {
    MlpChunk& C = M.chunk[k];
    if (!C.done) CK(cudaEventCreateWithFlags(&C.done, cudaEventDisableTiming));
    const size_t ny = (size_t)chunk * no;
    if (C.y.n < ny * E) CK(C.y.alloc(ny * E));
    if (C.mean.n < ny) CK(C.mean.alloc(ny));
    if (y_std && C.std.n < ny) CK(C.std.alloc(ny));
    if (C.spread.n < chunk) CK(C.spread.alloc(chunk));
  }
  auto submit = [&](uint64_t r0) -> int32_t {
    MlpChunk& C = M.chunk[(r0 / chunk) & 1u];
    const uint32_t rows = (uint32_t)std::min<uint64_t>(chunk, n - r0);
    if (r0 % group == 0)
      CK(cudaMemcpyAsync(M.xin.p, x + r0 * ni, std::min<uint64_t>(n - r0, group) * ni * 4, cudaMemcpyHostToDevice, s));
    MlpRowsArgs a{};
    a.net = M.net;
    a.rows = rows;
    a.P = M.P.p;
    a.img = M.img.p;
    a.X = M.xin.p + (r0 % group) * ni;
    a.x_mean = M.d_x_mean.p;
    a.x_sd = M.d_x_std.p;
    a.out = C.y.p;
    a.err = M.err.p;
    CK(launch_mlp_rows(a, E, false, s));
    CK(launch_mlp_ensemble(C.y.p, E, rows, no, M.d_y_mean.p, M.d_y_std.p, level, C.mean.p, y_std ? C.std.p : nullptr,
                           row_spread ? C.spread.p : nullptr, s));
    if (small) {
      float* h = M.h_small.p;
      CK(cudaMemcpyAsync(h, C.mean.p, n_mean * 4, cudaMemcpyDeviceToHost, s));
      if (n_std) CK(cudaMemcpyAsync(h + n_mean, C.std.p, n_std * 4, cudaMemcpyDeviceToHost, s));
      if (n_spread) CK(cudaMemcpyAsync(h + n_mean + n_std, C.spread.p, n_spread * 4, cudaMemcpyDeviceToHost, s));
    }
    if (r0 + rows == n) CK(fetch_err(M, s));
    CK(cudaEventRecord(C.done, s));
    return OMG_OK;
  };
  int32_t rc = OMG_OK;
  if ((rc = submit(0))) return rc;
  for (uint64_t r0 = 0; r0 < n; r0 += chunk) {
    if (n - r0 > chunk && (rc = submit(r0 + chunk))) return rc;
    if (r0 == 0) {
      populate_pages(y_mean, (size_t)n * no * 4);
      populate_pages(y_std, (size_t)n * no * 4);
    }
    MlpChunk& C = M.chunk[(r0 / chunk) & 1u];
    const uint64_t rows = std::min<uint64_t>(chunk, n - r0);
    if ((rc = wait_event(ctx, C.done, timeout_of(ctx)))) return rc;
    if (small) {
      const float* h = M.h_small.p;
      std::memcpy(y_mean, h, n_mean * 4);
      if (n_std) std::memcpy(y_std, h + n_mean, n_std * 4);
      if (n_spread) std::memcpy(row_spread, h + n_mean + n_std, n_spread * 4);
      break;
    }
    CK(cudaMemcpyAsync(y_mean + r0 * no, C.mean.p, rows * no * 4, cudaMemcpyDeviceToHost, M.back));
    if (y_std) CK(cudaMemcpyAsync(y_std + r0 * no, C.std.p, rows * no * 4, cudaMemcpyDeviceToHost, M.back));
    if (row_spread) CK(cudaMemcpyAsync(row_spread + r0, C.spread.p, rows * 4, cudaMemcpyDeviceToHost, M.back));
    CK(cudaStreamSynchronize(M.back));   // the chunk's buffers are free for the one after next
  }
  return check_err(ctx, M);
}

}  // namespace

extern "C" {

int32_t omg_surrogate_predict(omg_ctx* ctx, uint32_t id, const float* x, uint32_t n, float* y_mean, float* y_std) {
  return surrogate_run(ctx, id, x, n, y_mean, y_std, nullptr, 0.0f);
}

int32_t omg_surrogate_query(omg_ctx* ctx, uint32_t id, const float* x, uint32_t n, float* y_mean,
                            float* row_spread, float level) {
  if (!row_spread) return OMG_E_INVALID;
  return surrogate_run(ctx, id, x, n, y_mean, nullptr, row_spread, level);
}

// One forward/backward of `member` on standardized inputs and targets: the
// loss and the gradients of every layer (W row-major, then b), in order.
int32_t omg_mlp_grad(omg_ctx* ctx, uint32_t id, uint32_t member, const float* x, const float* y, uint32_t n,
                     float* loss, float* grads) {
  if (!ctx || !x || !y || n == 0 || n % 128 != 0) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  if (member >= M.cfg.members) return OMG_E_INVALID;
  int32_t rc = ensure_scratch(ctx, M, M.grad_s, n / 128u);
  if (rc) return rc;
  cudaStream_t s = ctx->stream;
  const MlpNet& N = M.net;
  if (M.grad_x.n < (size_t)n * M.cfg.n_in) CK(M.grad_x.alloc((size_t)n * M.cfg.n_in));
  if (M.grad_y.n < (size_t)n * M.cfg.n_out) CK(M.grad_y.alloc((size_t)n * M.cfg.n_out));
  CK(cudaMemcpyAsync(M.grad_x.p, x, (size_t)n * M.cfg.n_in * 4, cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(M.grad_y.p, y, (size_t)n * M.cfg.n_out * 4, cudaMemcpyHostToDevice, s));
  float* G = M.G.p + (uint64_t)member * N.p_stride;
  CK(cudaMemsetAsync(G, 0, (size_t)N.p_stride * 4, s));
  CK(cudaMemsetAsync(M.loss.p + member, 0, 4, s));
  CK(launch_mlp_rows(rows_args(M, M.grad_s, M.grad_x.p, M.grad_y.p, n, member), 1, true, s));
  CK(launch_mlp_dw(dw_args(M, M.grad_s, n, 1, member), ctx->n_sms, s));
  CK(cudaMemcpyAsync(M.h_loss.p, M.loss.p + member, 4, cudaMemcpyDeviceToHost, s));
  CK(fetch_err(M, s));
  uint64_t packed = 0;
  each_param(N, [&](uint32_t, uint32_t k) { packed += k; });
  if (grads && packed == N.p_stride) {
    CK(cudaMemcpyAsync(grads, G, packed * 4, cudaMemcpyDeviceToHost, s));   // the block has no padding
  } else if (grads) {
    cudaError_t e = cudaSuccess;
    uint64_t off = 0;
    each_param(N, [&](uint32_t at, uint32_t k) {
      if (e == cudaSuccess) e = cudaMemcpyAsync(grads + off, G + at, (size_t)k * 4, cudaMemcpyDeviceToHost, s);
      off += k;
    });
    CK(e);
  }
  CK(cudaStreamSynchronize(s));
  if (loss) *loss = M.h_loss.p[0];
  return check_err(ctx, M);
}

// Parameters: what = 1: standardization (x mean, x std, y mean, y std) then
// every member's layers (W row-major, b); what = 2: the AdamW moments (mW, vW,
// mb, vb per layer per member) then the step count. out = null: count only.
int32_t omg_mlp_params(omg_ctx* ctx, uint32_t id, uint32_t what, float* out, uint64_t* count) {
  if (!ctx || !count || (what != 1 && what != 2)) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  uint64_t n = 0;
  auto put_host = [&](const std::vector<float>& v) {
    if (out) std::copy(v.begin(), v.end(), out + n);
    n += v.size();
  };
  CK(cudaStreamSynchronize(ctx->stream));
  const MlpNet& N = M.net;
  const size_t np = (size_t)N.p_stride * N.members;
  std::vector<float> w, v;
  if (out) {
    w.resize(np);
    CK(cudaMemcpy(w.data(), what == 1 ? M.P.p : M.M1.p, np * 4, cudaMemcpyDeviceToHost));
    if (what == 2) {
      v.resize(np);
      CK(cudaMemcpy(v.data(), M.V1.p, np * 4, cudaMemcpyDeviceToHost));
    }
  }
  auto put = [&](const std::vector<float>& src, uint32_t e, uint32_t at, uint32_t k) {
    if (out) std::memcpy(out + n, src.data() + (size_t)e * N.p_stride + at, (size_t)k * 4);
    n += k;
  };
  if (what == 1) {
    put_host(M.x_mean);
    put_host(M.x_std);
    put_host(M.y_mean);
    put_host(M.y_std);
    for (uint32_t e = 0; e < N.members; e++) each_param(N, [&](uint32_t at, uint32_t k) { put(w, e, at, k); });
  } else {
    for (uint32_t e = 0; e < N.members; e++)
      for (uint32_t l = 0; l < N.n_layers; l++) {
        const MlpLayerDesc& D = N.L[l];
        put(w, e, D.w_off, D.in * D.out);
        put(v, e, D.w_off, D.in * D.out);
        put(w, e, D.b_off, D.out);
        put(v, e, D.b_off, D.out);
      }
    if (out) out[n] = (float)M.step;
    n += 1;
  }
  *count = n;
  return OMG_OK;
}

int32_t omg_mlp_set_params(omg_ctx* ctx, uint32_t id, uint32_t what, const float* in, uint64_t count) {
  if (!ctx || !in || (what != 1 && what != 2)) return OMG_E_INVALID;
  auto it = ctx->mlps.find(id);
  if (it == ctx->mlps.end()) return OMG_E_NOT_FOUND;
  MlpRec& M = *it->second;
  uint64_t need = 0;
  int32_t rc = omg_mlp_params(ctx, id, what, nullptr, &need);
  if (rc) return rc;
  if (count != need) return OMG_E_INVALID;
  uint64_t n = 0;
  auto get_host = [&](std::vector<float>& v) {
    std::copy(in + n, in + n + v.size(), v.begin());
    n += v.size();
  };
  const MlpNet& N = M.net;
  const size_t np = (size_t)N.p_stride * N.members;
  std::vector<float> w(np, 0.0f), v;
  auto get = [&](std::vector<float>& dst, uint32_t e, uint32_t at, uint32_t k) {
    std::memcpy(dst.data() + (size_t)e * N.p_stride + at, in + n, (size_t)k * 4);
    n += k;
  };
  if (what == 1) {
    get_host(M.x_mean);
    get_host(M.x_std);
    get_host(M.y_mean);
    get_host(M.y_std);
    for (uint32_t e = 0; e < N.members; e++) each_param(N, [&](uint32_t at, uint32_t k) { get(w, e, at, k); });
    CK(cudaMemcpy(M.P.p, w.data(), np * 4, cudaMemcpyHostToDevice));
    CK(launch_mlp_images(N, M.P.p, M.img.p, ctx->stream));
    int32_t rc2 = sync_norm(ctx, M);
    if (rc2) return rc2;
  } else {
    v.assign(np, 0.0f);
    for (uint32_t e = 0; e < N.members; e++)
      for (uint32_t l = 0; l < N.n_layers; l++) {
        const MlpLayerDesc& D = N.L[l];
        get(w, e, D.w_off, D.in * D.out);
        get(v, e, D.w_off, D.in * D.out);
        get(w, e, D.b_off, D.out);
        get(v, e, D.b_off, D.out);
      }
    CK(cudaMemcpy(M.M1.p, w.data(), np * 4, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(M.V1.p, v.data(), np * 4, cudaMemcpyHostToDevice));
    M.step = (uint64_t)in[n];
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return OMG_OK;
}

// Device time of the tensor-core GEMM at one shape, for the record: A [m x k]
// and B [n x k] bf16 (K-major), C f32 (atomically accumulated when k_split >
// 1), operands resident on the device; `reps` launches between two events on
// the context's stream after 3 untimed ones. *ms = mean per launch.
int32_t omg_tc_gemm_bench(omg_ctx* ctx, uint32_t m, uint32_t n, uint32_t k, uint32_t k_split, uint32_t reps,
                          float* ms) {
  if (!ctx || !ms || m == 0 || n == 0 || k == 0 || k % 8 != 0 || reps == 0 || k_split == 0 || k_split > 64)
    return OMG_E_INVALID;
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(ctx, cudaGetLastError(), "cudaSetDevice");
  cudaStream_t s = ctx->stream;
  DevBuf<uint16_t> da, db;
  DevBuf<float> dc;
  DevBuf<uint32_t> err;
  CK(da.alloc((size_t)m * k));
  CK(db.alloc((size_t)n * k));
  CK(dc.alloc((size_t)m * n));
  CK(err.alloc(1));
  CK(cudaMemsetAsync(err.p, 0, 4, s));
  CK(cudaMemsetAsync(da.p, 0x3C, (size_t)m * k * 2, s));   // bf16 0x3C3C (about 0.0115) everywhere
  CK(cudaMemsetAsync(db.p, 0x3C, (size_t)n * k * 2, s));
  CK(cudaMemsetAsync(dc.p, 0, (size_t)m * n * 4, s));
  GemmArgs g{};
  g.A = da.p;
  g.a_rs = k;
  g.a_ks = 1;
  g.B = db.p;
  g.b_rs = k;
  g.b_ks = 1;
  g.M = m;
  g.N = n;
  g.K = k;
  g.n_tile = n > 128 ? 128u : ((n + 15) & ~15u);
  g.D = dc.p;
  g.ldd = n;
  g.accumulate = k_split > 1 ? 1u : 0u;
  g.err = err.p;
  for (int i = 0; i < 3; i++) CK(launch_gemm(g, k_split, s));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  CK(cudaEventRecord(e0, s));
  for (uint32_t i = 0; i < reps; i++) CK(launch_gemm(g, k_split, s));
  CK(cudaEventRecord(e1, s));
  CK(cudaEventSynchronize(e1));
  float t = 0.0f;
  CK(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  uint32_t e = 0;
  CK(cudaMemcpy(&e, err.p, 4, cudaMemcpyDeviceToHost));
  if (e) {
    ctx->last_error = "tensor-core GEMM: an mbarrier wait ran out";
    return OMG_E_TIMEOUT;
  }
  *ms = t / (float)reps;
  return OMG_OK;
}

// The tensor-core GEMM alone: C[M x N] (f32) = A[M x K] . B[N x K]^T, A and B
// given as bf16 bit patterns in host memory (row-major, K contiguous).
int32_t omg_tc_gemm(omg_ctx* ctx, const uint16_t* a, const uint16_t* b, float* c, uint32_t m, uint32_t n,
                    uint32_t k) {
  if (!ctx || !a || !b || !c || m == 0 || n == 0 || k == 0) return OMG_E_INVALID;
  cudaStream_t s = ctx->stream;
  DevBuf<uint16_t> da, db;
  DevBuf<float> dc;
  DevBuf<uint32_t> err;
  CK(da.alloc((size_t)m * k));
  CK(db.alloc((size_t)n * k));
  CK(dc.alloc((size_t)m * n));
  CK(err.alloc(1));
  CK(cudaMemsetAsync(err.p, 0, 4, s));
  CK(cudaMemcpyAsync(da.p, a, (size_t)m * k * 2, cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(db.p, b, (size_t)n * k * 2, cudaMemcpyHostToDevice, s));
  GemmArgs g{};
  g.A = da.p;
  g.a_rs = k;
  g.a_ks = 1;
  g.B = db.p;
  g.b_rs = k;
  g.b_ks = 1;
  g.M = m;
  g.N = n;
  g.K = k;
  g.n_tile = n <= 256 ? ((n + 15) & ~15u) : 256;
  g.D = dc.p;
  g.ldd = n;
  g.err = err.p;
  CK(launch_gemm(g, 1, s));
  uint32_t e = 0;
  CK(cudaMemcpyAsync(c, dc.p, (size_t)m * n * 4, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(&e, err.p, 4, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (e) {
    ctx->last_error = "tensor-core GEMM: an mbarrier wait ran out";
    return OMG_E_TIMEOUT;
  }
  return OMG_OK;
}

}  // extern "C"
