// Host interface of the single-GPU fused kernels (no torch dependency).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace fairring {

struct AdamWArgs {
  float lr;
  float beta1;
  float beta2;
  float eps;
  float weight_decay;
  float step_size;       // lr / (1 - beta1^t)
  float inv_sqrt_bias2;  // 1 / sqrt(1 - beta2^t)
  float grad_scale;      // multiplied into the gradient first (clipping, loss scale)
};

// p, g, m, v: fp32, 16-byte aligned, n elements each.  Decoupled weight decay,
// same update as torch.optim.AdamW.
// shadow_bf16 (may be null): receives a bf16 copy of the updated parameters.
cudaError_t launchAdamWFlat(float* p, const float* g, float* m, float* v, void* shadow_bf16,
                            int64_t n, const AdamWArgs& a, int sm_count, cudaStream_t stream);
// dst (fp32, 16-byte aligned) = or += src (bf16, 16-byte aligned), n elements.
cudaError_t launchBf16GradToF32(float* dst, const void* src_bf16, int64_t n, bool accumulate,
                                int sm_count, cudaStream_t stream);
// *out = sum(x^2), or its square root; `partial`: scratch of sumSqBlocks(n, sm_count) floats,
// `done`: of one word.
int sumSqBlocks(int64_t n, int sm_count);
cudaError_t launchSumSq(const float* x, int64_t n, float* partial, unsigned* done, float* out, bool root,
                        int sm_count, cudaStream_t stream);

// Device-to-device copy by a kernel of at most `blocks` blocks (falls back to
// cudaMemcpyAsync when a pointer is not 16-byte aligned).
cudaError_t launchCopy(void* dst, const void* src, size_t bytes, int blocks, cudaStream_t stream);

// LayerNorm over the last dimension (`cols`, a multiple of 8, at most 8192) of a
// [rows, cols] tensor; x / dx are fp32 or bf16, y / dy are fp32 or bf16, the
// affine parameters and the saved per-row mean and 1/std are fp32.
cudaError_t launchLayerNormForward(const void* x, bool x_bf16, const float* gamma, const float* beta,
                                   void* y, bool y_bf16, float* mean, float* rstd, int64_t rows,
                                   int cols, float eps, int sm_count, cudaStream_t stream);
// `partial`: scratch of layerNormBackwardBlocks(rows, sm_count) x 2 x cols floats.
int layerNormBackwardBlocks(int64_t rows, int sm_count);
cudaError_t launchLayerNormBackward(const void* dy, bool y_bf16, const void* x, bool x_bf16,
                                    const float* gamma, const float* mean, const float* rstd, void* dx,
                                    float* partial, float* dgamma, float* dbeta, int64_t rows, int cols,
                                    int sm_count, cudaStream_t stream);

// xnew = x + branch (x fp32, branch fp32 or bf16), y = LayerNorm(xnew); the
// backward takes the gradient of y in its dtype and of an fp32 copy of it (`dy`,
// `dy32`: one may be null), adds `gres` (gradient arriving at xnew along the residual path, may
// be null) to the LayerNorm gradient and can also write the sum in bf16
// (`dbranch_bf16`, may be null).
cudaError_t launchAddLayerNormForward(const float* x, const void* branch, bool branch_bf16,
                                      const float* gamma, const float* beta, float* xnew, void* y,
                                      bool y_bf16, float* mean, float* rstd, int64_t rows, int cols,
                                      float eps, int sm_count, cudaStream_t stream);
cudaError_t launchAddLayerNormBackward(const void* dy, bool y_bf16, const float* dy32, const float* xnew,
                                       const float* gres, const float* gamma, const float* mean, const float* rstd,
                                       float* dx, void* dbranch_bf16, float* partial, float* dgamma,
                                       float* dbeta, int64_t rows, int cols, int sm_count,
                                       cudaStream_t stream);

// out = x + branch: n elements (a multiple of 8), the branch bf16, 16-byte aligned.
cudaError_t launchAddBranch(const float* x, const void* branch_bf16, float* out, int64_t n, cudaStream_t stream);

// Softmax cross-entropy over [rows, vocab] logits (fp32 or bf16): per-row loss
// and log-sum-exp (2 x rows: rounded, and what the rounding cut off); the row of a target that is negative or past the vocabulary has
// loss 0; with `classes` > 0 a target is an error unless it is below that or -100.
cudaError_t launchCrossEntropyForward(const void* logits, bool bf16, const int64_t* targets, float* loss,
                                      float* lse, int64_t rows, int vocab, int classes, cudaStream_t stream);
// *mean = sum of `loss` / *count, *count = max(number of targets >= 0, least).
cudaError_t launchCrossEntropyMean(const float* loss, const int64_t* targets, int64_t rows, float least,
                                   float* mean, float* count, cudaStream_t stream);
// The gradient, scaled by *upstream / *count * scale (device scalars, count may be
// null); `grad` may be the logits themselves and lies as they do relative to a
// 16-byte boundary.
cudaError_t launchCrossEntropyBackward(const void* logits, void* grad, bool bf16, const int64_t* targets,
                                       const float* lse, const float* upstream, const float* count, float scale,
                                       int64_t rows, int vocab, cudaStream_t stream);

// Training-mode BatchNorm of a channels-last tensor, [rows = N*H*W, channels], fp32
// or bf16, `channels` a power of two from 8 to 2048, more than one row; the
// affine parameters and statistics are fp32.  All tensors 16-byte aligned.
struct BatchNormShape {
  int64_t rows;
  int channels;
};
int batchNormParts(const BatchNormShape& s, int sm_count);
int64_t batchNormScratchFloats(const BatchNormShape& s, int sm_count);
// y = BatchNorm(x) [+ residual] [, ReLU]; writes the batch's mean and 1/std, moves
// the running statistics (variance with n - 1) and counts the batch in *tracked.
cudaError_t launchBatchNormForward(const BatchNormShape& s, bool bf16, const void* x, const void* residual, void* y,
                                   bool relu, const float* gamma, const float* beta, float* mean, float* rstd,
                                   float* running_mean, float* running_var, int64_t* tracked, float momentum,
                                   float eps, float* scratch, int sm_count, cudaStream_t stream);
// `y`, `dz`: given when there was a residual and a ReLU: the output, and where the
// residual's gradient goes.  Without a ReLU the residual's gradient is dy.  `dy2` (may be null,
// only then): a second gradient of y, added to dy.
cudaError_t launchBatchNormBackward(const BatchNormShape& s, bool bf16, const void* dy, const void* dy2, const void* x,
                                    const void* y, void* dz, void* dx, bool relu, const float* gamma, const float* beta,
                                    const float* mean, const float* rstd, float* dgamma, float* dbeta,
                                    float* scratch, int sm_count, cudaStream_t stream);

// y = GELU(x) of n bf16 elements (a multiple of 8), tanh or erf form; 16-byte aligned.
cudaError_t launchGeluForward(const void* x, void* y, int64_t n, bool tanh_form, cudaStream_t stream);
// out[c] (fp32 or bf16) = sum over the rows of a [rows, cols] bf16 matrix, cols a multiple of
// 8: of dy or, with `gelu_x`, of dx = dy * GELU'(gelu_x), which is written.  `partial`:
// scratch of columnSumStrips(rows, cols, sm_count) x cols floats.
int columnSumStrips(int64_t rows, int cols, int sm_count);
cudaError_t launchColumnSum(const void* dy, const void* gelu_x, bool tanh_form, void* dx, float* partial, void* out,
                            bool out_bf16, int64_t rows, int cols, int sm_count, cudaStream_t stream);

// Max pooling of a channels-last tensor, fp32 or bf16, channels a multiple of 8, square windows of at
// most 16 x 16; all tensors 16-byte aligned.  `chosen`: one byte per output element, the position of
// the largest element in its window.
struct PoolShape {
  int images, channels, in_h, in_w, out_h, out_w, window, stride, pad;
};
cudaError_t launchMaxPoolForward(const PoolShape& s, bool bf16, const void* x, void* y, void* chosen,
                                 cudaStream_t stream);
cudaError_t launchMaxPoolBackward(const PoolShape& s, bool bf16, const void* dy, const void* chosen, void* dx,
                                  cudaStream_t stream);

// x[b][s] = table[tokens[b][s]] + pos[s], rows of d floats (a multiple of 4), 16-byte aligned.
cudaError_t launchEmbedForward(const int64_t* tokens, const float* table, const float* pos, float* x, int batch, int seq,
                               int64_t vocab, int d, cudaStream_t stream);
// dtable[tokens[b][s]] += dx[b][s]; dpos[s] = sum over b of dx[b][s].  The order of the additions depends on
// the tokens and the sizes alone.
cudaError_t launchEmbedBackward(const float* dx, const int64_t* tokens, float* dtable, float* dpos, int batch, int seq,
                                int64_t vocab, int d, int sm_count, cudaStream_t stream);

// Channels-last [images, 3, height, width] (fp32 or bf16) to channels-last bf16 [images, 16, rows, cols]:
// the 2 x 2 pixel blocks from row and column -4 on, 4 x 3 channels and 4 zeros; zero outside the image.
cudaError_t launchStemFold(const void* image, bool bf16, void* out, int images, int height, int width, int rows,
                           int cols, cudaStream_t stream);

uint64_t localLaunchCountImpl();
void noteLocalLaunch();

}  // namespace fairring
