#include "local_ops.h"

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <optional>
#include <tuple>

#include "kernels/local_kernels.h"

namespace fairring {

namespace {
void checkFlat(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous(), name,
              " must be a contiguous fp32 CUDA tensor");
}

// The tensor itself where its memory starts on a 16-byte boundary, else a copy that does.
at::Tensor aligned16(const at::Tensor& t) {
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone();
}

// A sum over rows that a kernel will write, or zeros where there is no row and no launch.
at::Tensor sumOfRows(int64_t rows, at::IntArrayRef sizes, const at::TensorOptions& options) {
  return rows > 0 ? at::empty(sizes, options) : at::zeros(sizes, options);
}

// One AdamW step over flat buffers, in place.  `step` counts from 1.
void adamwFlat(at::Tensor p, at::Tensor g, at::Tensor m, at::Tensor v, double lr, double beta1,
               double beta2, double eps, double weight_decay, int64_t step, double grad_scale,
               c10::optional<at::Tensor> shadow) {
  checkFlat(p, "param");
  checkFlat(g, "grad");
  checkFlat(m, "exp_avg");
  checkFlat(v, "exp_avg_sq");
  TORCH_CHECK(g.numel() == p.numel() && m.numel() == p.numel() && v.numel() == p.numel(),
              "flat buffers must have the same length");
  TORCH_CHECK(step >= 1, "step counts from 1");
  void* shadow_ptr = nullptr;
  if (shadow.has_value() && shadow->defined()) {
    TORCH_CHECK(shadow->is_cuda() && shadow->scalar_type() == at::kBFloat16 &&
                    shadow->is_contiguous() && shadow->numel() == p.numel(),
                "shadow must be a contiguous bf16 CUDA tensor as long as param");
    shadow_ptr = shadow->data_ptr();
  }
  c10::cuda::CUDAGuard guard(p.device());
  AdamWArgs a;
  a.lr = (float)lr;
  a.beta1 = (float)beta1;
  a.beta2 = (float)beta2;
  a.eps = (float)eps;
  a.weight_decay = (float)weight_decay;
  a.step_size = (float)(lr / (1.0 - std::pow(beta1, (double)step)));
  a.inv_sqrt_bias2 = (float)(1.0 / std::sqrt(1.0 - std::pow(beta2, (double)step)));
  a.grad_scale = (float)grad_scale;
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  cudaError_t e = launchAdamWFlat(p.data_ptr<float>(), g.data_ptr<float>(), m.data_ptr<float>(),
                                  v.data_ptr<float>(), shadow_ptr, p.numel(), a, sms,
                                  c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "adamw_flat launch failed: ", cudaGetErrorString(e));
}

// dst (fp32) = or += src (bf16); both contiguous, same length.
void bf16GradToF32(at::Tensor dst, at::Tensor src, bool accumulate) {
  TORCH_CHECK(dst.is_cuda() && dst.scalar_type() == at::kFloat && dst.is_contiguous(),
              "dst must be a contiguous fp32 CUDA tensor");
  TORCH_CHECK(src.is_cuda() && src.scalar_type() == at::kBFloat16 && src.is_contiguous() &&
                  src.numel() == dst.numel(),
              "src must be a contiguous bf16 CUDA tensor as long as dst");
  c10::cuda::CUDAGuard guard(dst.device());
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  cudaError_t e = launchBf16GradToF32(dst.data_ptr<float>(), src.data_ptr(), dst.numel(), accumulate,
                                      sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "bf16_grad_to_f32 launch failed: ", cudaGetErrorString(e));
}

// Sum of squares of a flat fp32 buffer, or its square root, as a 1-element device tensor.
at::Tensor sumSq(at::Tensor x, bool root) {
  checkFlat(x, "input");
  c10::cuda::CUDAGuard guard(x.device());
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  const int blocks = sumSqBlocks(x.numel(), sms);
  at::Tensor out = at::empty({1}, x.options()), scratch = at::empty({blocks + 1}, x.options());
  float* partial = scratch.data_ptr<float>();
  cudaError_t e = launchSumSq(x.data_ptr<float>(), x.numel(), partial, reinterpret_cast<unsigned*>(partial + blocks),
                              out.data_ptr<float>(), root, sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "sumsq launch failed: ", cudaGetErrorString(e));
  return out;
}

// y, mean, rstd = layer_norm(x); y in `out_dtype` (fp32 or bf16).
std::tuple<at::Tensor, at::Tensor, at::Tensor> layerNormForward(at::Tensor x, at::Tensor gamma,
                                                                at::Tensor beta, double eps,
                                                                at::ScalarType out_dtype) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.dim() >= 1, "x must be a contiguous CUDA tensor");
  TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16, "x must be fp32 or bf16");
  TORCH_CHECK(out_dtype == at::kFloat || out_dtype == at::kBFloat16, "output must be fp32 or bf16");
  const int64_t cols = x.size(-1);
  const int64_t rows = x.numel() / std::max<int64_t>(cols, 1);
  TORCH_CHECK(gamma.is_cuda() && beta.is_cuda() && gamma.scalar_type() == at::kFloat &&
                  beta.scalar_type() == at::kFloat && gamma.is_contiguous() && beta.is_contiguous() &&
                  gamma.numel() == cols && beta.numel() == cols,
              "weight and bias must be contiguous fp32 CUDA vectors of the row length");
  TORCH_CHECK(cols % 8 == 0 && cols <= 8192, "row length must be a multiple of 8, at most 8192");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  gamma = aligned16(gamma);
  beta = aligned16(beta);
  at::Tensor y = at::empty(x.sizes(), x.options().dtype(out_dtype));
  at::Tensor mean = at::empty({rows}, x.options().dtype(at::kFloat));
  at::Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  cudaError_t e = launchLayerNormForward(
      x.data_ptr(), x.scalar_type() == at::kBFloat16, gamma.data_ptr<float>(), beta.data_ptr<float>(),
      y.data_ptr(), out_dtype == at::kBFloat16, mean.data_ptr<float>(), rstd.data_ptr<float>(), rows,
      (int)cols, (float)eps, sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "layer_norm forward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(y, mean, rstd);
}

// dx, dgamma, dbeta
std::tuple<at::Tensor, at::Tensor, at::Tensor> layerNormBackward(at::Tensor dy, at::Tensor x,
                                                                 at::Tensor gamma, at::Tensor mean,
                                                                 at::Tensor rstd) {
  TORCH_CHECK(dy.is_cuda() && dy.is_contiguous() && x.is_contiguous() && dy.sizes() == x.sizes(),
              "dy and x must be contiguous and equally shaped");
  TORCH_CHECK(dy.scalar_type() == at::kFloat || dy.scalar_type() == at::kBFloat16, "dy must be fp32 or bf16");
  const int64_t cols = x.size(-1);
  const int64_t rows = x.numel() / std::max<int64_t>(cols, 1);
  c10::cuda::CUDAGuard guard(x.device());
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  dy = aligned16(dy);
  x = aligned16(x);
  gamma = aligned16(gamma);
  at::Tensor dx = at::empty_like(x);
  at::Tensor dgamma = sumOfRows(rows, {cols}, gamma.options());
  at::Tensor dbeta = sumOfRows(rows, {cols}, gamma.options());
  at::Tensor partial = at::empty({(int64_t)layerNormBackwardBlocks(rows, sms), 2, cols}, gamma.options());
  cudaError_t e = launchLayerNormBackward(
      dy.data_ptr(), dy.scalar_type() == at::kBFloat16, x.data_ptr(), x.scalar_type() == at::kBFloat16,
      gamma.data_ptr<float>(), mean.data_ptr<float>(), rstd.data_ptr<float>(), dx.data_ptr(),
      partial.data_ptr<float>(), dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), rows, (int)cols, sms,
      c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "layer_norm backward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(dx, dgamma, dbeta);
}

// xnew, y, mean, rstd = x + branch, layer_norm(x + branch); x fp32, branch fp32 or bf16.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> addLayerNormForward(
    at::Tensor x, at::Tensor branch, at::Tensor gamma, at::Tensor beta, double eps,
    at::ScalarType out_dtype) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.scalar_type() == at::kFloat && x.dim() >= 1,
              "x must be a contiguous fp32 CUDA tensor");
  TORCH_CHECK(branch.is_cuda() && branch.is_contiguous() && branch.sizes() == x.sizes() &&
                  (branch.scalar_type() == at::kFloat || branch.scalar_type() == at::kBFloat16),
              "branch must be contiguous, shaped like x, fp32 or bf16");
  TORCH_CHECK(out_dtype == at::kFloat || out_dtype == at::kBFloat16, "output must be fp32 or bf16");
  const int64_t cols = x.size(-1);
  const int64_t rows = x.numel() / std::max<int64_t>(cols, 1);
  TORCH_CHECK(gamma.is_cuda() && beta.is_cuda() && gamma.scalar_type() == at::kFloat &&
                  beta.scalar_type() == at::kFloat && gamma.is_contiguous() && beta.is_contiguous() &&
                  gamma.numel() == cols && beta.numel() == cols,
              "weight and bias must be contiguous fp32 CUDA vectors of the row length");
  TORCH_CHECK(cols % 8 == 0 && cols <= 8192, "row length must be a multiple of 8, at most 8192");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  branch = aligned16(branch);
  gamma = aligned16(gamma);
  beta = aligned16(beta);
  at::Tensor xnew = at::empty_like(x);
  at::Tensor y = at::empty(x.sizes(), x.options().dtype(out_dtype));
  at::Tensor mean = at::empty({rows}, x.options());
  at::Tensor rstd = at::empty({rows}, x.options());
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  cudaError_t e = launchAddLayerNormForward(
      x.data_ptr<float>(), branch.data_ptr(), branch.scalar_type() == at::kBFloat16, gamma.data_ptr<float>(),
      beta.data_ptr<float>(), xnew.data_ptr<float>(), y.data_ptr(), out_dtype == at::kBFloat16,
      mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, (int)cols, (float)eps, sms,
      c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "add_layer_norm forward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(xnew, y, mean, rstd);
}

// x + branch in fp32, x fp32 and the branch bf16.
at::Tensor addBranch(at::Tensor x, at::Tensor branch) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.scalar_type() == at::kFloat && branch.is_cuda() &&
                  branch.device() == x.device() && branch.is_contiguous() && branch.scalar_type() == at::kBFloat16 &&
                  branch.sizes() == x.sizes() && x.numel() % 8 == 0,
              "x must be contiguous fp32, branch contiguous bf16 and shaped alike, a multiple of 8 elements");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  branch = aligned16(branch);
  at::Tensor out = at::empty_like(x);
  cudaError_t e = launchAddBranch(x.data_ptr<float>(), branch.data_ptr(), out.data_ptr<float>(), x.numel(),
                                  c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "residual add launch failed: ", cudaGetErrorString(e));
  return out;
}

// dx (fp32), dx in bf16 (or an undefined tensor), dgamma, dbeta.  `dy`: the gradient
// of y, `dy32`: of its fp32 copy (one may be missing); `gres`: the gradient that
// reaches xnew along the residual path, or nothing.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> addLayerNormBackward(
    std::optional<at::Tensor> dy, at::Tensor xnew, at::Tensor gamma, at::Tensor mean, at::Tensor rstd,
    std::optional<at::Tensor> gres, bool want_bf16, std::optional<at::Tensor> dy32) {
  TORCH_CHECK(xnew.is_cuda() && xnew.is_contiguous() && xnew.scalar_type() == at::kFloat,
              "xnew must be a contiguous fp32 CUDA tensor");
  c10::cuda::CUDAGuard guard(xnew.device());
  auto given = [&](const std::optional<at::Tensor>& t, const char* name, bool fp32) -> at::Tensor {
    if (!t.has_value() || !t->defined()) return {};
    TORCH_CHECK(t->is_cuda() && t->is_contiguous() && t->sizes() == xnew.sizes() &&
                    (t->scalar_type() == at::kFloat || (!fp32 && t->scalar_type() == at::kBFloat16)),
                name, " must be contiguous, shaped like xnew, fp32", fp32 ? "" : " or bf16");
    return aligned16(*t);
  };
  const at::Tensor d = given(dy, "dy", false), d32 = given(dy32, "dy32", true), res = given(gres, "gres", true);
  TORCH_CHECK(d.defined() || d32.defined(), "one of dy and dy32 is needed");
  xnew = aligned16(xnew);
  gamma = aligned16(gamma);
  const int64_t cols = xnew.size(-1);
  const int64_t rows = xnew.numel() / std::max<int64_t>(cols, 1);
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  at::Tensor dx = at::empty_like(xnew);
  at::Tensor dbr;
  if (want_bf16) dbr = at::empty(xnew.sizes(), xnew.options().dtype(at::kBFloat16));
  at::Tensor dgamma = sumOfRows(rows, {cols}, gamma.options());
  at::Tensor dbeta = sumOfRows(rows, {cols}, gamma.options());
  at::Tensor partial = at::empty({(int64_t)layerNormBackwardBlocks(rows, sms), 2, cols}, gamma.options());
  cudaError_t e = launchAddLayerNormBackward(
      d.defined() ? d.data_ptr() : nullptr, d.defined() && d.scalar_type() == at::kBFloat16,
      d32.defined() ? d32.data_ptr<float>() : nullptr, xnew.data_ptr<float>(),
      res.defined() ? res.data_ptr<float>() : nullptr, gamma.data_ptr<float>(), mean.data_ptr<float>(),
      rstd.data_ptr<float>(), dx.data_ptr<float>(), want_bf16 ? dbr.data_ptr() : nullptr, partial.data_ptr<float>(),
      dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), rows, (int)cols, sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "add_layer_norm backward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(dx, dbr, dgamma, dbeta);
}

void checkBf16Matrix(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.scalar_type() == at::kBFloat16 && t.dim() >= 1 &&
                  t.size(-1) % 8 == 0 && t.size(-1) > 0 && t.size(-1) <= INT32_MAX,
              name, " must be a contiguous bf16 CUDA tensor whose last dimension is a multiple of 8");
}

at::Tensor geluForward(at::Tensor x, bool tanh_form) {
  checkBf16Matrix(x, "x");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  at::Tensor y = at::empty_like(x);
  cudaError_t e = launchGeluForward(x.data_ptr(), y.data_ptr(), x.numel(), tanh_form,
                                    c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "gelu forward launch failed: ", cudaGetErrorString(e));
  return y;
}

// Column sums of dy or, with `gelu_x`, of dx = dy * gelu'(gelu_x), in `out_dtype`; and dx.
std::tuple<at::Tensor, at::Tensor> columnSumOf(at::Tensor dy, std::optional<at::Tensor> gelu_x, bool tanh_form,
                                               at::ScalarType out_dtype) {
  checkBf16Matrix(dy, "dy");
  TORCH_CHECK(out_dtype == at::kFloat || out_dtype == at::kBFloat16, "the sums are fp32 or bf16");
  c10::cuda::CUDAGuard guard(dy.device());
  dy = aligned16(dy);
  at::Tensor x, dx;
  if (gelu_x.has_value()) {
    checkBf16Matrix(*gelu_x, "x");
    TORCH_CHECK(gelu_x->sizes() == dy.sizes() && gelu_x->device() == dy.device(), "x and dy must be equally shaped");
    x = aligned16(*gelu_x);
    dx = at::empty_like(dy);
  }
  const int64_t cols = dy.size(-1), rows = dy.numel() / cols;
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  at::Tensor out = at::empty({cols}, dy.options().dtype(out_dtype));
  at::Tensor partial = at::empty({(int64_t)columnSumStrips(rows, (int)cols, sms), cols}, dy.options().dtype(at::kFloat));
  cudaError_t e = launchColumnSum(dy.data_ptr(), x.defined() ? x.data_ptr() : nullptr, tanh_form,
                                  dx.defined() ? dx.data_ptr() : nullptr, partial.data_ptr<float>(), out.data_ptr(),
                                  out_dtype == at::kBFloat16, rows, (int)cols, sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "column sum launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(dx, out);
}

at::Tensor columnSum(at::Tensor dy, at::ScalarType out_dtype) {
  return std::get<1>(columnSumOf(dy, std::nullopt, false, out_dtype));
}

std::tuple<at::Tensor, at::Tensor> geluBackward(at::Tensor dy, at::Tensor x, bool tanh_form, at::ScalarType sum_dtype) {
  return columnSumOf(dy, x, tanh_form, sum_dtype);
}

void checkLogits(const at::Tensor& logits, const at::Tensor& targets) {
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.is_contiguous(),
              "logits must be a contiguous 2-D CUDA tensor");
  TORCH_CHECK(logits.scalar_type() == at::kFloat || logits.scalar_type() == at::kBFloat16,
              "logits must be fp32 or bf16");
  TORCH_CHECK(targets.is_cuda() && targets.device() == logits.device() && targets.scalar_type() == at::kLong &&
                  targets.is_contiguous() && targets.numel() == logits.size(0),
              "targets must be a contiguous int64 CUDA vector with one entry per row");
  TORCH_CHECK(logits.size(1) > 0 && logits.size(1) <= INT32_MAX, "the vocabulary must not be empty");
}

// (per-row loss, [2, rows] log-sum-exp and what its rounding cut off) of logits [rows, vocab] against targets [rows];
// `classes`, if not 0: a target that is neither one of them nor -100 is an error.
std::tuple<at::Tensor, at::Tensor> crossEntropyForward(at::Tensor logits, at::Tensor targets, int64_t classes) {
  checkLogits(logits, targets);
  TORCH_CHECK(classes >= 0 && classes <= logits.size(1), "no more classes than logits");
  c10::cuda::CUDAGuard guard(logits.device());
  auto fopt = logits.options().dtype(at::kFloat);
  at::Tensor loss = at::empty({logits.size(0)}, fopt), lse = at::empty({2, logits.size(0)}, fopt);
  cudaError_t e = launchCrossEntropyForward(logits.data_ptr(), logits.scalar_type() == at::kBFloat16,
                                            targets.data_ptr<int64_t>(), loss.data_ptr<float>(),
                                            lse.data_ptr<float>(), logits.size(0), (int)logits.size(1),
                                            (int)classes, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "cross_entropy forward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(loss, lse);
}

// (mean loss over the rows whose target is not negative, how many those are, at least `least`)
std::tuple<at::Tensor, at::Tensor> crossEntropyMean(at::Tensor losses, at::Tensor targets, double least) {
  checkFlat(losses, "losses");
  TORCH_CHECK(targets.is_cuda() && targets.device() == losses.device() && targets.scalar_type() == at::kLong &&
                  targets.is_contiguous() && targets.numel() == losses.numel(),
              "targets must be a contiguous int64 CUDA vector with one entry per row");
  c10::cuda::CUDAGuard guard(losses.device());
  at::Tensor mean = at::empty({}, losses.options()), count = at::empty({1}, losses.options());
  cudaError_t e = launchCrossEntropyMean(losses.data_ptr<float>(), targets.data_ptr<int64_t>(), losses.numel(),
                                         (float)least, mean.data_ptr<float>(), count.data_ptr<float>(),
                                         c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "cross_entropy mean launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(mean, count);
}

// Writes d(loss)/d(logits) * upstream / count * scale to `grad`, which may be the logits.
void crossEntropyBackward(at::Tensor grad, at::Tensor logits, at::Tensor targets, at::Tensor lse, at::Tensor upstream,
                          double scale, std::optional<at::Tensor> count) {
  checkLogits(logits, targets);
  TORCH_CHECK(grad.is_cuda() && grad.device() == logits.device() && grad.is_contiguous() &&
                  grad.sizes() == logits.sizes() && grad.scalar_type() == logits.scalar_type(),
              "grad must be like the logits");
  TORCH_CHECK(lse.is_cuda() && lse.scalar_type() == at::kFloat && lse.is_contiguous() &&
                  lse.numel() == 2 * logits.size(0),
              "lse must be the contiguous fp32 [2, rows] CUDA tensor that the forward made");
  TORCH_CHECK(upstream.is_cuda() && upstream.scalar_type() == at::kFloat && upstream.numel() == 1,
              "upstream must be a one-element fp32 CUDA tensor");
  const float* count_ptr = nullptr;
  if (count.has_value() && count->defined()) {
    TORCH_CHECK(count->is_cuda() && count->scalar_type() == at::kFloat && count->numel() == 1,
                "count must be a one-element fp32 CUDA tensor");
    count_ptr = count->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(logits.device());
  cudaError_t e = launchCrossEntropyBackward(
      logits.data_ptr(), grad.data_ptr(), logits.scalar_type() == at::kBFloat16, targets.data_ptr<int64_t>(),
      lse.data_ptr<float>(), upstream.data_ptr<float>(), count_ptr, (float)scale, logits.size(0),
      (int)logits.size(1), c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "cross_entropy backward launch failed: ", cudaGetErrorString(e));
}

void crossEntropyBackwardInPlace(at::Tensor logits, at::Tensor targets, at::Tensor lse, at::Tensor upstream,
                                 double scale, std::optional<at::Tensor> count) {
  crossEntropyBackward(logits, logits, targets, lse, upstream, scale, count);
}

BatchNormShape batchNormShape(const at::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4 && x.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                  (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16),
              "x must be a channels-last fp32 or bf16 CUDA tensor");
  const int64_t c = x.size(1);
  TORCH_CHECK(c >= 8 && c <= 2048 && (c & (c - 1)) == 0, "channels must be a power of two from 8 to 2048");
  TORCH_CHECK(x.numel() / c > 1, "more than one value per channel is needed");
  return {x.numel() / c, (int)c};
}

void checkLikeX(const at::Tensor& t, const at::Tensor& x, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.device() == x.device() && t.scalar_type() == x.scalar_type() &&
                  t.sizes() == x.sizes() && t.is_contiguous(at::MemoryFormat::ChannelsLast),
              name, " must be like x: device, type, shape, channels-last");
}

void checkPerChannel(const at::Tensor& t, const at::Tensor& x, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.device() == x.device() && t.scalar_type() == at::kFloat && t.is_contiguous() &&
                  t.numel() == x.size(1) && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0,
              name, " must be a contiguous, 16-byte aligned fp32 CUDA vector with one entry per channel");
}

// y, mean, rstd of training-mode BatchNorm [+ residual] [, ReLU]; moves the running statistics.
std::tuple<at::Tensor, at::Tensor, at::Tensor> batchNormForward(
    at::Tensor x, std::optional<at::Tensor> residual, at::Tensor gamma, at::Tensor beta, at::Tensor running_mean,
    at::Tensor running_var, at::Tensor tracked, double momentum, double eps, bool relu) {
  const BatchNormShape s = batchNormShape(x);
  checkPerChannel(gamma, x, "weight");
  checkPerChannel(beta, x, "bias");
  checkPerChannel(running_mean, x, "running_mean");
  checkPerChannel(running_var, x, "running_var");
  TORCH_CHECK(tracked.is_cuda() && tracked.device() == x.device() && tracked.scalar_type() == at::kLong &&
                  tracked.numel() == 1,
              "num_batches_tracked must be one int64 on the GPU");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  at::Tensor res;
  if (residual.has_value() && residual->defined()) {
    checkLikeX(*residual, x, "residual");
    res = aligned16(*residual);
  }
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  auto fopt = x.options().dtype(at::kFloat).memory_format(at::MemoryFormat::Contiguous);
  at::Tensor y = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  at::Tensor mean = at::empty({s.channels}, fopt), rstd = at::empty({s.channels}, fopt);
  at::Tensor scratch = at::empty({batchNormScratchFloats(s, sms)}, fopt);
  cudaError_t e = launchBatchNormForward(
      s, x.scalar_type() == at::kBFloat16, x.data_ptr(), res.defined() ? res.data_ptr() : nullptr, y.data_ptr(), relu,
      gamma.data_ptr<float>(), beta.data_ptr<float>(), mean.data_ptr<float>(), rstd.data_ptr<float>(),
      running_mean.data_ptr<float>(), running_var.data_ptr<float>(), tracked.data_ptr<int64_t>(), (float)momentum,
      (float)eps, scratch.data_ptr<float>(), sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "batch_norm forward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(y, mean, rstd);
}

// dx, gradient of the residual, dgamma, dbeta.  `y`: the output, given when there
// was a residual and a ReLU; otherwise the second result is undefined.  `dy2`: a second gradient of
// that output, or nothing.
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> batchNormBackward(
    at::Tensor dy, at::Tensor x, std::optional<at::Tensor> y, at::Tensor gamma, at::Tensor beta, at::Tensor mean,
    at::Tensor rstd, bool relu, std::optional<at::Tensor> dy2) {
  const BatchNormShape s = batchNormShape(x);
  checkLikeX(dy, x, "dy");
  checkPerChannel(gamma, x, "weight");
  checkPerChannel(beta, x, "bias");
  checkPerChannel(mean, x, "mean");
  checkPerChannel(rstd, x, "rstd");
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  dy = aligned16(dy);
  at::Tensor second;
  if (dy2.has_value() && dy2->defined()) {
    checkLikeX(*dy2, x, "dy2");
    second = aligned16(*dy2);
  }
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  at::Tensor dz, yt;
  if (y.has_value() && y->defined()) {
    checkLikeX(*y, x, "y");
    yt = aligned16(*y);
    dz = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  }
  at::Tensor dx = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  at::Tensor dgamma = at::empty_like(gamma), dbeta = at::empty_like(gamma);
  at::Tensor scratch = at::empty({batchNormScratchFloats(s, sms)}, gamma.options());
  cudaError_t e = launchBatchNormBackward(
      s, x.scalar_type() == at::kBFloat16, dy.data_ptr(), second.defined() ? second.data_ptr() : nullptr, x.data_ptr(),
      yt.defined() ? yt.data_ptr() : nullptr,
      dz.defined() ? dz.data_ptr() : nullptr, dx.data_ptr(), relu, gamma.data_ptr<float>(), beta.data_ptr<float>(),
      mean.data_ptr<float>(), rstd.data_ptr<float>(), dgamma.data_ptr<float>(), dbeta.data_ptr<float>(),
      scratch.data_ptr<float>(), sms, c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "batch_norm backward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(dx, dz, dgamma, dbeta);
}

PoolShape poolShape(const at::Tensor& x, int64_t window, int64_t stride, int64_t pad) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4 && x.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                  (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16) && x.size(1) % 8 == 0 &&
                  x.numel() > 0,
              "x must be a channels-last fp32 or bf16 CUDA tensor whose channels are a multiple of 8");
  TORCH_CHECK(window >= 1 && window <= 16 && stride >= 1 && pad >= 0 && 2 * pad <= window &&
                  x.size(2) + 2 * pad >= window && x.size(3) + 2 * pad >= window && x.numel() / 8 < INT32_MAX,
              "the window does not fit");
  const int64_t oh = (x.size(2) + 2 * pad - window) / stride + 1, ow = (x.size(3) + 2 * pad - window) / stride + 1;
  return {(int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)oh, (int)ow, (int)window, (int)stride,
          (int)pad};
}

// y and, one byte per element of it, which element of the window it is.
std::tuple<at::Tensor, at::Tensor> maxPoolForward(at::Tensor x, int64_t window, int64_t stride, int64_t pad) {
  const PoolShape s = poolShape(x, window, stride, pad);
  c10::cuda::CUDAGuard guard(x.device());
  x = aligned16(x);
  const at::Tensor y = at::empty({s.images, s.channels, s.out_h, s.out_w}, x.options(), at::MemoryFormat::ChannelsLast);
  const at::Tensor chosen = at::empty({y.numel()}, x.options().dtype(at::kByte));
  cudaError_t e = launchMaxPoolForward(s, x.scalar_type() == at::kBFloat16, x.data_ptr(), y.data_ptr(),
                                       chosen.data_ptr(), c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "max_pool forward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(y, chosen);
}

at::Tensor maxPoolBackward(at::Tensor dy, at::Tensor x, at::Tensor chosen, int64_t window, int64_t stride, int64_t pad) {
  const PoolShape s = poolShape(x, window, stride, pad);
  TORCH_CHECK(dy.is_cuda() && dy.device() == x.device() && dy.scalar_type() == x.scalar_type() && dy.dim() == 4 &&
                  dy.size(0) == s.images && dy.size(1) == s.channels && dy.size(2) == s.out_h &&
                  dy.size(3) == s.out_w && dy.is_contiguous(at::MemoryFormat::ChannelsLast),
              "dy must be channels-last and shaped like the output");
  TORCH_CHECK(chosen.is_cuda() && chosen.scalar_type() == at::kByte && chosen.is_contiguous() &&
                  chosen.numel() == dy.numel(),
              "chosen must hold one byte per output element");
  c10::cuda::CUDAGuard guard(x.device());
  dy = aligned16(dy);
  const at::Tensor dx = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  cudaError_t e = launchMaxPoolBackward(s, x.scalar_type() == at::kBFloat16, dy.data_ptr(), chosen.data_ptr(),
                                        dx.data_ptr(), c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "max_pool backward launch failed: ", cudaGetErrorString(e));
  return dx;
}

void checkTokens(const at::Tensor& tokens, int64_t positions) {
  TORCH_CHECK(tokens.is_cuda() && tokens.dim() == 2 && tokens.scalar_type() == at::kLong && tokens.is_contiguous() &&
                  tokens.numel() < INT32_MAX && tokens.size(1) <= positions,
              "tokens must be a contiguous [batch, sequence] int64 CUDA tensor, no longer than the positions");
}

// table[tokens] + pos[0..sequence), fp32.
at::Tensor embedForward(at::Tensor tokens, at::Tensor table, at::Tensor pos) {
  for (const at::Tensor& t : {table, pos})
    TORCH_CHECK(t.is_cuda() && t.device() == tokens.device() && t.dim() == 2 && t.scalar_type() == at::kFloat &&
                    t.is_contiguous() && t.size(1) == table.size(1) && t.size(1) % 8 == 0 &&
                    reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0,
                "the tables must be contiguous, 16-byte aligned fp32 CUDA matrices of equal width, a multiple of 8");
  checkTokens(tokens, pos.size(0));
  c10::cuda::CUDAGuard guard(tokens.device());
  at::Tensor x = at::empty({tokens.size(0), tokens.size(1), table.size(1)}, table.options());
  cudaError_t e = launchEmbedForward(tokens.data_ptr<int64_t>(), table.data_ptr<float>(), pos.data_ptr<float>(),
                                     x.data_ptr<float>(), (int)tokens.size(0), (int)tokens.size(1), table.size(0),
                                     (int)table.size(1), c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "embedding forward launch failed: ", cudaGetErrorString(e));
  return x;
}

// Gradients of the table and of the positions: `dx` reached the lookup, `dlow` (bf16) the
// table's bf16 copy; either may be missing.
std::tuple<at::Tensor, at::Tensor> embedBackward(std::optional<at::Tensor> dx, std::optional<at::Tensor> dlow,
                                                 at::Tensor tokens, int64_t vocab, int64_t positions, int64_t d) {
  checkTokens(tokens, positions);
  c10::cuda::CUDAGuard guard(tokens.device());
  auto fopt = tokens.options().dtype(at::kFloat);
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  const auto stream = c10::cuda::getCurrentCUDAStream();
  at::Tensor dtable;
  if (dlow.has_value() && dlow->defined()) {
    TORCH_CHECK(dlow->is_cuda() && dlow->device() == tokens.device() && dlow->scalar_type() == at::kBFloat16 &&
                    dlow->is_contiguous() && dlow->dim() == 2 && dlow->size(0) == vocab && dlow->size(1) == d,
                "dlow must be a contiguous bf16 matrix shaped like the table");
    const at::Tensor low = aligned16(*dlow);
    dtable = at::empty({vocab, d}, fopt);
    cudaError_t e = launchBf16GradToF32(dtable.data_ptr<float>(), low.data_ptr(), dtable.numel(), false, sms, stream);
    TORCH_CHECK(e == cudaSuccess, "embedding backward launch failed: ", cudaGetErrorString(e));
  } else {
    dtable = at::zeros({vocab, d}, fopt);
  }
  if (!dx.has_value() || !dx->defined()) return std::make_tuple(dtable, at::zeros({positions, d}, fopt));
  TORCH_CHECK(dx->is_cuda() && dx->device() == tokens.device() && dx->scalar_type() == at::kFloat &&
                  dx->is_contiguous() && dx->numel() == tokens.numel() * d && d % 8 == 0,
              "dx must be contiguous fp32 with one row per token");
  const at::Tensor g = aligned16(*dx);
  at::Tensor dpos = sumOfRows(tokens.size(1) < positions ? 0 : tokens.numel(), {positions, d}, fopt);
  cudaError_t e = launchEmbedBackward(g.data_ptr<float>(), tokens.data_ptr<int64_t>(), dtable.data_ptr<float>(),
                                      dpos.data_ptr<float>(), (int)tokens.size(0), (int)tokens.size(1), vocab, (int)d, sms,
                                      stream);
  TORCH_CHECK(e == cudaSuccess, "embedding backward launch failed: ", cudaGetErrorString(e));
  return std::make_tuple(dtable, dpos);
}

// The folded input of a 7 x 7, stride 2, padding 3 convolution over 3 channels.
at::Tensor stemFold(at::Tensor image) {
  TORCH_CHECK(image.is_cuda() && image.dim() == 4 && image.size(1) == 3 && image.numel() > 0 &&
                  image.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                  (image.scalar_type() == at::kFloat || image.scalar_type() == at::kBFloat16),
              "the image must be a channels-last fp32 or bf16 CUDA tensor of 3 channels");
  c10::cuda::CUDAGuard guard(image.device());
  const int64_t rows = (image.size(2) + 1) / 2 + 3, cols = (image.size(3) + 1) / 2 + 3;
  TORCH_CHECK(image.size(0) * rows * cols <= INT32_MAX, "the image is too large");
  at::Tensor out = at::empty({image.size(0), 16, rows, cols}, image.options().dtype(at::kBFloat16),
                             at::MemoryFormat::ChannelsLast);
  cudaError_t e = launchStemFold(image.data_ptr(), image.scalar_type() == at::kBFloat16, out.data_ptr(),
                                 (int)image.size(0), (int)image.size(2), (int)image.size(3), (int)rows, (int)cols,
                                 c10::cuda::getCurrentCUDAStream());
  TORCH_CHECK(e == cudaSuccess, "stem fold launch failed: ", cudaGetErrorString(e));
  return out;
}

// ---- autograd nodes ------------------------------------------------------------
// LayerNorm and the loss as native nodes: one call from Python forward and none backward.  For
// 777 x 4104 rows the kernels take 27 us of a pass that took 110 us with Python nodes.
// Where the graph of a backward is itself wanted, it is made of torch's ops (the two functions below).
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// dx, dgamma, dbeta of LayerNorm, differentiable.
std::tuple<at::Tensor, at::Tensor, at::Tensor> layerNormBackwardGraph(const at::Tensor& dy, const at::Tensor& x,
                                                                      const at::Tensor& gamma, const at::Tensor& mean,
                                                                      const at::Tensor& rstd) {
  const at::Tensor g = dy.to(at::kFloat);
  const auto [dx, dgamma, unused] = at::native_layer_norm_backward(g, x.to(at::kFloat), {x.size(-1)}, mean, rstd, gamma,
                                                                   std::nullopt, {true, true, false});
  return std::make_tuple(dx.to(x.scalar_type()), dgamma, g.reshape({-1, x.size(-1)}).sum(0));
}

// The gradient of the mean cross-entropy, differentiable; the logits stay as they are.
at::Tensor crossEntropyBackwardGraph(const at::Tensor& logits, const at::Tensor& targets, const at::Tensor& upstream,
                                     const at::Tensor& count) {
  const at::Tensor counts = targets.ge(0).logical_and(targets.lt(logits.size(1))).unsqueeze(1);
  const at::Tensor at = at::where(counts, targets.unsqueeze(1), at::zeros_like(targets).unsqueeze(1));
  const at::Tensor p = at::softmax(logits.to(at::kFloat), 1);
  const at::Tensor d = p - at::zeros_like(p).scatter_(1, at, 1.0);
  const at::Tensor grad = at::where(counts, d * (upstream.to(at::kFloat) / count), at::zeros_like(p));
  return grad.to(logits.scalar_type());
}

struct LayerNormNode : torch::autograd::Function<LayerNormNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& gamma, const at::Tensor& beta,
                            double eps, at::ScalarType out_dtype) {
    auto [y, mean, rstd] = layerNormForward(x, gamma, beta, eps, out_dtype);
    ctx->save_for_backward({x, gamma, mean, rstd});
    ctx->saved_data["out"] = static_cast<int64_t>(out_dtype);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    if (at::GradMode::is_enabled()) {
      auto [dx, dgamma, dbeta] = layerNormBackwardGraph(grads[0], saved[0], saved[1], saved[2], saved[3]);
      return {dx, dgamma, dbeta, at::Tensor(), at::Tensor()};
    }
    const at::Tensor dy = grads[0].to(static_cast<at::ScalarType>(ctx->saved_data["out"].toInt())).contiguous();
    auto [dx, dgamma, dbeta] = layerNormBackward(dy, saved[0], saved[1], saved[2], saved[3]);
    return {dx, dgamma, dbeta, at::Tensor(), at::Tensor()};
  }
};

// (x + branch, LayerNorm(x + branch)); the gradient that reaches the sum along the residual path is
// added inside the LayerNorm's backward kernel, and the result goes to both addends.
struct AddLayerNormNode : torch::autograd::Function<AddLayerNormNode> {
  static variable_list forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& branch,
                               const at::Tensor& gamma, const at::Tensor& beta, double eps, at::ScalarType out_dtype) {
    auto [xnew, y, mean, rstd] = addLayerNormForward(x.contiguous(), branch.contiguous(), gamma, beta, eps, out_dtype);
    ctx->set_materialize_grads(false);  // an unused output arrives undefined, not as zeros
    ctx->save_for_backward({xnew, gamma, mean, rstd});
    ctx->saved_data["out"] = static_cast<int64_t>(out_dtype);
    ctx->saved_data["branch"] = static_cast<int64_t>(branch.scalar_type());
    return {xnew, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &xnew = saved[0], &gamma = saved[1];
    const auto branch_dtype = static_cast<at::ScalarType>(ctx->saved_data["branch"].toInt());
    if (!grads[1].defined()) {  // the normalised output was not used: only the residual path carries gradient
      const at::Tensor g = grads[0].defined() ? grads[0] : at::zeros_like(xnew);
      return {g, g.to(branch_dtype), at::zeros_like(gamma), at::zeros_like(gamma), at::Tensor(), at::Tensor()};
    }
    if (at::GradMode::is_enabled()) {  // xnew, an output of this node, carries the graph of both addends
      auto [dx, dgamma, dbeta] = layerNormBackwardGraph(grads[1], xnew, gamma, saved[2], saved[3]);
      if (grads[0].defined()) dx = dx + grads[0];
      return {dx, dx.to(branch_dtype), dgamma, dbeta, at::Tensor(), at::Tensor()};
    }
    const at::Tensor dy = grads[1].to(static_cast<at::ScalarType>(ctx->saved_data["out"].toInt())).contiguous();
    std::optional<at::Tensor> gres;
    if (grads[0].defined()) gres = grads[0].to(at::kFloat).contiguous();
    const bool want_bf16 = branch_dtype == at::kBFloat16;
    auto [dx, dbr, dgamma, dbeta] =
        addLayerNormBackward(dy, xnew, gamma, saved[2], saved[3], gres, want_bf16, std::nullopt);
    return {dx, want_bf16 ? dbr : dx, dgamma, dbeta, at::Tensor(), at::Tensor()};
  }
};

// Mean cross-entropy.  `classes` > 0: as torch's own loss -- the logits stay as they are (they may be more
// than the classes), no counted row gives NaN, a target that is no class is an error unless it is -100; otherwise the gradient is written over the logits.
struct CrossEntropyNode : torch::autograd::Function<CrossEntropyNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& logits, const at::Tensor& targets, int64_t classes) {
    const bool keep = classes > 0;
    auto [losses, lse] = crossEntropyForward(logits, targets, classes);
    auto [mean, count] = crossEntropyMean(losses, targets, keep ? 0.0 : 1.0);
    ctx->save_for_backward({logits, targets, lse, count});
    ctx->saved_data["keep"] = keep;
    return mean;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &logits = saved[0], &targets = saved[1];
    const bool keep = ctx->saved_data["keep"].toBool();
    if (at::GradMode::is_enabled())
      return {crossEntropyBackwardGraph(logits, targets, grads[0], saved[3]), at::Tensor(), at::Tensor()};
    const at::Tensor grad = keep ? at::empty_like(logits) : logits.detach();
    crossEntropyBackward(grad, logits, targets, saved[2], grads[0].to(at::kFloat).reshape({1}), 1.0, saved[3]);
    return {grad, at::Tensor(), at::Tensor()};
  }
};

at::Tensor layerNorm(const at::Tensor& x, const at::Tensor& gamma, const at::Tensor& beta, double eps,
                     at::ScalarType out_dtype) {
  return LayerNormNode::apply(x.contiguous(), gamma, beta, eps, out_dtype);
}
std::tuple<at::Tensor, at::Tensor> addLayerNorm(const at::Tensor& x, const at::Tensor& branch, const at::Tensor& gamma,
                                                const at::Tensor& beta, double eps, at::ScalarType out_dtype) {
  auto out = AddLayerNormNode::apply(x, branch, gamma, beta, eps, out_dtype);
  return std::make_tuple(out[0], out[1]);
}
at::Tensor crossEntropy(const at::Tensor& logits, const at::Tensor& targets, int64_t classes) {
  return CrossEntropyNode::apply(logits, targets, classes);
}
}  // namespace

uint64_t localLaunchCount() { return localLaunchCountImpl(); }

void bindLocalOps(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("adamw_flat_", &adamwFlat, py::arg("param"), py::arg("grad"), py::arg("exp_avg"),
        py::arg("exp_avg_sq"), py::arg("lr"), py::arg("beta1"), py::arg("beta2"), py::arg("eps"),
        py::arg("weight_decay"), py::arg("step"), py::arg("grad_scale") = 1.0,
        py::arg("shadow") = py::none());
  m.def("bf16_grad_to_f32_", &bf16GradToF32, py::arg("dst"), py::arg("src"),
        py::arg("accumulate") = false);
  m.def("layer_norm", &layerNorm, py::arg("x"), py::arg("weight"), py::arg("bias"), py::arg("eps"),
        py::arg("out_dtype"));
  m.def("add_layer_norm", &addLayerNorm, py::arg("x"), py::arg("branch"), py::arg("weight"), py::arg("bias"),
        py::arg("eps"), py::arg("out_dtype"));
  m.def("cross_entropy", &crossEntropy, py::arg("logits"), py::arg("targets"), py::arg("classes") = 0);
  m.def("layer_norm_bwd_graph", &layerNormBackwardGraph, py::arg("dy"), py::arg("x"), py::arg("weight"),
        py::arg("mean"), py::arg("rstd"));
  m.def("cross_entropy_bwd_graph", &crossEntropyBackwardGraph, py::arg("logits"), py::arg("targets"),
        py::arg("upstream"), py::arg("count"));
  m.def("sumsq", &sumSq, py::arg("x"), py::arg("root") = false);
  m.def("cross_entropy_fwd", &crossEntropyForward, py::arg("logits"), py::arg("targets"),
        py::arg("classes") = 0);
  m.def("cross_entropy_mean", &crossEntropyMean, py::arg("losses"), py::arg("targets"), py::arg("least"));
  m.def("cross_entropy_bwd", &crossEntropyBackward, py::arg("grad"), py::arg("logits"), py::arg("targets"),
        py::arg("lse"), py::arg("upstream"), py::arg("scale"), py::arg("count") = py::none());
  m.def("cross_entropy_bwd_", &crossEntropyBackwardInPlace, py::arg("logits"), py::arg("targets"),
        py::arg("lse"), py::arg("upstream"), py::arg("scale"), py::arg("count") = py::none());
  m.def("add_layer_norm_fwd", &addLayerNormForward, py::arg("x"), py::arg("branch"), py::arg("weight"),
        py::arg("bias"), py::arg("eps"), py::arg("out_dtype"));
  m.def("add_branch", &addBranch, py::arg("x"), py::arg("branch"));
  m.def("add_layer_norm_bwd", &addLayerNormBackward, py::arg("dy"), py::arg("xnew"), py::arg("weight"),
        py::arg("mean"), py::arg("rstd"), py::arg("gres"), py::arg("want_bf16"), py::arg("dy32") = py::none());
  m.def("gelu_fwd", &geluForward, py::arg("x"), py::arg("tanh_form"));
  m.def("gelu_bwd", &geluBackward, py::arg("dy"), py::arg("x"), py::arg("tanh_form"), py::arg("sum_dtype"));
  m.def("column_sum", &columnSum, py::arg("x"), py::arg("dtype"));
  m.def("batch_norm_fwd", &batchNormForward, py::arg("x"), py::arg("residual"), py::arg("weight"), py::arg("bias"),
        py::arg("running_mean"), py::arg("running_var"), py::arg("tracked"), py::arg("momentum"), py::arg("eps"),
        py::arg("relu"));
  m.def("batch_norm_bwd", &batchNormBackward, py::arg("dy"), py::arg("x"), py::arg("y"), py::arg("weight"),
        py::arg("bias"), py::arg("mean"), py::arg("rstd"), py::arg("relu"), py::arg("dy2") = py::none());
  m.def("max_pool_fwd", &maxPoolForward, py::arg("x"), py::arg("window"), py::arg("stride"), py::arg("pad"));
  m.def("max_pool_bwd", &maxPoolBackward, py::arg("dy"), py::arg("x"), py::arg("chosen"), py::arg("window"),
        py::arg("stride"), py::arg("pad"));
  m.def("embed_fwd", &embedForward, py::arg("tokens"), py::arg("table"), py::arg("pos"));
  m.def("embed_bwd", &embedBackward, py::arg("dx"), py::arg("dlow"), py::arg("tokens"), py::arg("vocab"),
        py::arg("positions"), py::arg("d"));
  m.def("stem_fold", &stemFold, py::arg("image"));
  m.def("layer_norm_fwd", &layerNormForward, py::arg("x"), py::arg("weight"), py::arg("bias"),
        py::arg("eps"), py::arg("out_dtype"));
  m.def("layer_norm_bwd", &layerNormBackward, py::arg("dy"), py::arg("x"), py::arg("weight"),
        py::arg("mean"), py::arg("rstd"));
}

}  // namespace fairring
