// The surrogate network's device layout and launches (mlp_net.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace omg {

constexpr uint32_t kMlpWide = 256;       // widest hidden or output layer
constexpr int kMlpMaxLayers = 17;

// One layer inside a member's parameter block (floats, offsets multiples of 4:
// W [out x in] row-major, then b) and inside its image block (bf16: the
// weights as 8 x 8 core matrices, ip x op with ip, op the sizes rounded up to
// 16 and zeros beyond in, out).
struct MlpLayerDesc {
  uint32_t in, out, ip, op;
  uint32_t w_off, b_off, img_off, pad;
};
struct MlpNet {
  uint32_t n_layers, members;
  uint32_t p_stride;                     // floats of one member (a multiple of 4)
  uint32_t img_stride;                   // bf16 elements of one member
  MlpLayerDesc L[kMlpMaxLayers];
};

struct MlpRowsArgs {
  MlpNet net;
  uint32_t rows;                         // rows of the batch (training: a multiple of 128)
  uint32_t member0;                      // first member of the launch
  const float* P;
  const uint16_t* img;
  const float* X;                        // [.. x in]: inference: raw, x_mean and x_sd apply; training: standardized
  const float *x_mean, *x_sd;
  float* out;                            // inference: [member][rows][out]
  // training: targets, the loss (added here), scratch per (member of the
  // launch, row tile): x image, hidden activation images, dZ images (128 x
  // kMlpWide slots per layer), GELU'(Z) per hidden layer, the bias gradients'
  // sums of 32 rows (4 x layers x kMlpWide)
  const float* Y;
  float* loss;
  uint16_t *xt, *at, *dzt;
  float *gz, *gb;
  // rows of X and Y of this step: perm[half of the step's epoch][member][step in epoch][row]; null: row i
  const uint32_t* perm;
  uint64_t perm_half, perm_member;
  const uint32_t* step;
  uint32_t spe;
  uint32_t* err;                         // error word: 16 = an mbarrier wait ran out
};
struct MlpDwArgs {
  MlpNet net;
  uint32_t tiles, members, member0;
  uint32_t shares, share_rows;           // set by launch_mlp_dw: the shares of the rows (dw_shares), and
  uint32_t group, group0;                // the shares that a CTA takes, and of the first layer
  float* G;
  const uint16_t *xt, *at, *dzt;
  const float* gb;
  uint32_t* err;
};
struct MlpAdamwArgs {
  MlpNet net;
  float *P, *M1, *V1, *G;
  uint16_t* img;
  const float* sched;                    // per step: learning rate, bias corrections 1 and 2
  uint32_t* step;
  uint32_t* ticket;
  float* loss;                           // [member], this step's; cleared
  float* epoch_loss;                     // [member][epochs]: the last step's loss of every epoch
  uint32_t spe, epochs;
  float b1, b2, eps, wd;
};

cudaError_t mlp_net_init();
cudaError_t launch_mlp_rows(const MlpRowsArgs& a, uint32_t members, bool train, cudaStream_t s);
// The shares of `rows` rows that a weight gradient is summed in, and a share's rows (the last has what is left).
uint32_t dw_shares(uint32_t rows, uint32_t& share_rows);
cudaError_t launch_mlp_dw(MlpDwArgs a, int n_sms, cudaStream_t s);
cudaError_t launch_mlp_adamw(const MlpAdamwArgs& a, cudaStream_t s);
cudaError_t launch_mlp_images(const MlpNet& net, const float* P, uint16_t* img, cudaStream_t s);
cudaError_t launch_mlp_ensemble(const float* y, uint32_t members, uint32_t rows, uint32_t cols, const float* mean,
                                const float* sd, float level, float* out_mean, float* out_std, float* out_spread,
                                cudaStream_t s);

}  // namespace omg
