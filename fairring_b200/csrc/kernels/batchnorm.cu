// Training-mode BatchNorm over channels-last activations with the ReLU and the
// residual add behind it (sm_100a), for the convolutional workload.
//
// A channels-last tensor is a [rows = N*H*W, channels] matrix.  Every kernel
// here is a stream over that matrix, bound by HBM: a thread owns the same 8
// channels (16 bytes of bf16) in every row it visits, so a block of 256 threads
// reads 4 KiB of contiguous memory at a time and the per-channel constants stay
// in registers.  This needs channels / 8 to divide the block: powers of two from
// 8 to 2048.  Passes over memory, bytes per bf16 element:
//   forward   statistics (read x: 2), apply (read x and the residual, write y: 4 or 6)
//   backward  sums (read dy and x: 4; with a residual also y, writing the masked
//             gradient: 8), dx (read gradient and x, write dx: 6)
// The ReLU's mask is recomputed from x where there is no residual; with one, the
// masked gradient is the residual's gradient, which has to be written anyway.
//
// Statistics: every thread sums differences from its own first element, turns
// them into (count, mean, M2), and these are merged over the block and then, in
// fp64, over the grid, so nothing cancels whatever the channel's mean is.
//
// ResNet-50, 256 images of 224 x 224 in bf16 (53 BatchNorms): torch's statistics,
// transform, reduction and gradient kernels took 31.4 ms of a step, its ReLU and add
// passes around them another 4.9 ms; the kernels here take 9.0 ms for all of it, at
// 4.5 to 6 TB/s in the large layers (a copy moves 6.5), and the step went from 54.3
// to 27.5 ms (22.3 ms with the later steps around it).
//
// The two small kernels between the passes read one partial result per block of
// the first pass: 8 channels and 128 results side by side, all of a thread's loads in
// flight (5.4 and 3.7 us on average; with 32 channels a block and up to 20 results a
// thread 10.6 and 7.5 us).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "local_kernels.h"
#include "vec8.cuh"

namespace fairring {
namespace {

constexpr int kBnThreads = 256;
// The small kernels: 8 channels (a 32-byte sector) and 128 partial results side by side.
constexpr int kBnFinishThreads = 1024;
constexpr int kBnFinishRows = kBnFinishThreads / 8;
constexpr int kBnFinishLoads = 5;
constexpr int kBnMaxBlocks = kBnFinishRows * kBnFinishLoads;

__device__ __forceinline__ void loadChannels(const float* p, int group, float (&v)[8]) {
  Raw8<float> r;
  r.load(p + group * 8);
  r.get(v);
}

// Vectors in flight per thread and stream: 64 bytes.
template <typename T> constexpr int kBnUnroll = sizeof(T) == 2 ? 4 : 2;

// part[block][0][c] = mean and part[block][1][c] = M2 of this block's rows; how
// many those are, the merge works out.
template <typename T>
__global__ void __launch_bounds__(kBnThreads, 4)
bn_stats_kernel(const T* __restrict__ x, int64_t nvec, int groups, float* __restrict__ part) {
  constexpr int U = kBnUnroll<T>;
  const int64_t stride = (int64_t)gridDim.x * kBnThreads;
  int64_t i = (int64_t)blockIdx.x * kBnThreads + threadIdx.x;
  float pivot[8] = {}, s[8] = {}, ss[8] = {};
  int n = 0;
  if (i < nvec) {
    Raw8<T> r;
    r.load(x + i * 8);
    r.get(pivot);
  }
  auto add = [&](const Raw8<T>& r) {
    float v[8];
    r.get(v);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float d = v[k] - pivot[k];
      s[k] += d;
      ss[k] = fmaf(d, d, ss[k]);
    }
    ++n;
  };
  for (; i + (U - 1) * stride < nvec; i += U * stride) {
    Raw8<T> r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) r[u].load(x + (i + u * stride) * 8);
#pragma unroll
    for (int u = 0; u < U; ++u) add(r[u]);
  }
  for (; i < nvec; i += stride) {
    Raw8<T> r;
    r.load(x + i * 8);
    add(r);
  }

  __shared__ float sm_mean[kBnThreads * 9], sm_m2[kBnThreads * 9], sm_n[kBnThreads];
  const float inv = n > 0 ? 1.f / n : 0.f;
  sm_n[threadIdx.x] = (float)n;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    sm_mean[threadIdx.x * 9 + k] = pivot[k] + s[k] * inv;
    sm_m2[threadIdx.x * 9 + k] = ss[k] - s[k] * s[k] * inv;
  }
  __syncthreads();
  const int channels = groups * 8, members = kBnThreads / groups;
  for (int c = threadIdx.x; c < channels; c += kBnThreads) {
    const int g = c >> 3, k = c & 7;
    const float first = sm_mean[g * 9 + k];
    float count = 0.f, d = 0.f;
    for (int m = 0; m < members; ++m) {
      const int t = m * groups + g;
      count += sm_n[t];
      d += sm_n[t] * (sm_mean[t * 9 + k] - first);
    }
    const float mean = first + (count > 0.f ? d / count : 0.f);
    float m2 = 0.f;
    for (int m = 0; m < members; ++m) {
      const int t = m * groups + g;
      const float e = sm_mean[t * 9 + k] - mean;
      m2 += sm_m2[t * 9 + k] + sm_n[t] * e * e;
    }
    part[(size_t)blockIdx.x * 2 * channels + c] = mean;
    part[((size_t)blockIdx.x * 2 + 1) * channels + c] = m2;
  }
}

// Sum over the block of what each thread holds for channel threadIdx.x % 8: warp w < 8
// gets channel w's.
__device__ __forceinline__ double sumOfChannel(double v, double (&sm)[kBnFinishThreads / 32][9]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  __syncthreads();
  if (lane < 8) sm[w][lane] = v;
  __syncthreads();
  double t = w < 8 ? sm[lane][w] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Merges the blocks' statistics, 8 channels per block, and updates the running ones.
// `members`: rows that a block of the first pass visits at a time.
__global__ void __launch_bounds__(kBnFinishThreads, 1)
bn_finish_stats_kernel(const float* __restrict__ part, int nparts, int members, int channels, int64_t rows,
                       float eps, float momentum, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                       float* __restrict__ running_mean, float* __restrict__ running_var,
                       int64_t* __restrict__ tracked) {
  __shared__ double sm[kBnFinishThreads / 32][9];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 8 + (threadIdx.x & 7), row = threadIdx.x >> 3;
  const float first = part[c];  // block 0's mean: what the others are merged around
  float mean[kBnFinishLoads], m2[kBnFinishLoads];
#pragma unroll
  for (int j = 0; j < kBnFinishLoads; ++j) {
    const int b = row + j * kBnFinishRows;
    mean[j] = b < nparts ? part[(size_t)b * 2 * channels + c] : 0.f;
    m2[j] = b < nparts ? part[((size_t)b * 2 + 1) * channels + c] : 0.f;
  }
  // Rows of block b: whole rounds of the grid, and its share of the last one.
  const int64_t round = (int64_t)nparts * members;
  const int whole = (int)(rows / round) * members, rest = (int)(rows % round);
  double d = 0.0, q = 0.0;
#pragma unroll
  for (int j = 0; j < kBnFinishLoads; ++j) {
    const int b = row + j * kBnFinishRows;
    if (b < nparts) {
      const double n = whole + min(members, max(0, rest - b * members)), e = (double)mean[j] - (double)first;
      d += n * e;
      q += (double)m2[j] + n * e * e;
    }
  }
  d = sumOfChannel(d, sm) / (double)rows;
  q = sumOfChannel(q, sm) / (double)rows;
  const int mine = blockIdx.x * 8 + w;
  if (lane == 0 && w < 8) {
    const float mu = (float)((double)part[mine] + d);
    double var = q - d * d;
    if (var < 0.0) var = 0.0;  // NaN stays
    mean_out[mine] = mu;
    rstd_out[mine] = rsqrtf((float)var + eps);
    running_mean[mine] = (1.f - momentum) * running_mean[mine] + momentum * mu;
    running_var[mine] =
        (1.f - momentum) * running_var[mine] + momentum * (float)(var * ((double)rows / (double)(rows - 1)));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *tracked += 1;
}

// y = (x - mean) * rstd * gamma + beta [+ residual] [, negative values to zero].  From
// the end to the start, as the dx pass below: the end of x is what the pass before
// left in L2 (2 to 3 % of either).
template <typename T, bool kRelu, bool kResidual>
__global__ void __launch_bounds__(kBnThreads, 4)
bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ residual, T* __restrict__ y,
                const float* __restrict__ mean, const float* __restrict__ rstd,
                const float* __restrict__ gamma, const float* __restrict__ beta, int64_t nvec, int groups) {
  constexpr int U = 2;
  const int group = threadIdx.x % groups;
  float mu[8], scale[8], shift[8];
  loadChannels(mean, group, mu);
  loadChannels(beta, group, shift);
  {
    float g[8];
    loadChannels(rstd, group, scale);
    loadChannels(gamma, group, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) scale[k] *= g[k];
  }
  const int64_t stride = (int64_t)gridDim.x * kBnThreads;
  auto one = [&](const Raw8<T>& rx, const Raw8<T>& rr, int64_t at) {
    float v[8], o[8];
    rx.get(v);
    if constexpr (kResidual) rr.get(o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float z = fmaf(v[k] - mu[k], scale[k], shift[k]);
      if constexpr (kResidual) z += o[k];
      if constexpr (kRelu) z = z < 0.f ? 0.f : z;  // NaN stays
      o[k] = z;
    }
    Raw8<T> out;
    out.set(o);
    out.store(y + at * 8);
  };
  const int64_t first = (int64_t)blockIdx.x * kBnThreads + threadIdx.x;
  int64_t i = first < nvec ? first + (nvec - 1 - first) / stride * stride : -1;  // the thread's last vector
  for (; i - (U - 1) * stride >= 0; i -= U * stride) {
    Raw8<T> rx[U], rr[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rx[u].load(x + (i - u * stride) * 8);
      if constexpr (kResidual) rr[u].load(residual + (i - u * stride) * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) one(rx[u], rr[u], i - u * stride);
  }
  for (; i >= 0; i -= stride) {
    Raw8<T> rx, rr;
    rx.load(x + i * 8);
    if constexpr (kResidual) rr.load(residual + i * 8);
    one(rx, rr, i);
  }
}

// How the gradient passes the ReLU.
enum BnMask { kBnNone, kBnFromX, kBnFromY };

// part[block][0][c] = sum dz, part[block][1][c] = sum dz * (x - mean), where dz is
// dy behind the mask; with kBnFromY dz is written out as well.  kTwo: the output was
// used twice, by the next convolution and as the next residual, and dy + dy2 is its
// gradient: adding them here costs 15 us where the pass that autograd would add them in
// took 74 us (means over ResNet-50's blocks, 256 images).
template <typename T, BnMask kMask, bool kTwo = false>
__global__ void __launch_bounds__(kBnThreads, 4)
bn_bwd_sums_kernel(const T* __restrict__ dy, const T* __restrict__ dy2, const T* __restrict__ x,
                   const T* __restrict__ y, T* __restrict__ dz, const float* __restrict__ mean, const float* __restrict__ rstd,
                   const float* __restrict__ gamma, const float* __restrict__ beta, int64_t nvec, int groups,
                   float* __restrict__ part) {
  constexpr int U = 2;
  const int group = threadIdx.x % groups;
  float mu[8], scale[8], shift[8], s1[8] = {}, s2[8] = {};
  loadChannels(mean, group, mu);
  if constexpr (kMask == kBnFromX) {
    float g[8];
    loadChannels(beta, group, shift);
    loadChannels(rstd, group, scale);
    loadChannels(gamma, group, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) scale[k] *= g[k];
  }
  const int64_t stride = (int64_t)gridDim.x * kBnThreads;
  auto one = [&](const Raw8<T>& rd, const Raw8<T>& rd2, const Raw8<T>& rx, const Raw8<T>& ry, int64_t at) {
    float d[8], v[8], o[8];
    rd.get(d);
    if constexpr (kTwo) {
      rd2.get(o);
#pragma unroll
      for (int k = 0; k < 8; ++k) d[k] += o[k];
    }
    rx.get(v);
    if constexpr (kMask == kBnFromY) ry.get(o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float e = v[k] - mu[k];
      if constexpr (kMask == kBnFromX) d[k] = fmaf(e, scale[k], shift[k]) <= 0.f ? 0.f : d[k];
      if constexpr (kMask == kBnFromY) d[k] = o[k] <= 0.f ? 0.f : d[k];
      s1[k] += d[k];
      s2[k] = fmaf(d[k], e, s2[k]);
    }
    if constexpr (kMask == kBnFromY) {
      Raw8<T> out;
      out.set(d);
      out.store(dz + at * 8);
    }
  };
  int64_t i = (int64_t)blockIdx.x * kBnThreads + threadIdx.x;
  for (; i + (U - 1) * stride < nvec; i += U * stride) {
    Raw8<T> rd[U], rd2[U], rx[U], ry[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rd[u].load(dy + (i + u * stride) * 8);
      if constexpr (kTwo) rd2[u].load(dy2 + (i + u * stride) * 8);
      rx[u].load(x + (i + u * stride) * 8);
      if constexpr (kMask == kBnFromY) ry[u].load(y + (i + u * stride) * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) one(rd[u], rd2[u], rx[u], ry[u], i + u * stride);
  }
  for (; i < nvec; i += stride) {
    Raw8<T> rd, rd2, rx, ry;
    rd.load(dy + i * 8);
    if constexpr (kTwo) rd2.load(dy2 + i * 8);
    rx.load(x + i * 8);
    if constexpr (kMask == kBnFromY) ry.load(y + i * 8);
    one(rd, rd2, rx, ry, i);
  }

  __shared__ float sm1[kBnThreads * 9], sm2[kBnThreads * 9];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    sm1[threadIdx.x * 9 + k] = s1[k];
    sm2[threadIdx.x * 9 + k] = s2[k];
  }
  __syncthreads();
  const int channels = groups * 8, members = kBnThreads / groups;
  for (int c = threadIdx.x; c < channels; c += kBnThreads) {
    const int g = c >> 3, k = c & 7;
    float a = 0.f, b = 0.f;
    for (int m = 0; m < members; ++m) {
      a += sm1[(m * groups + g) * 9 + k];
      b += sm2[(m * groups + g) * 9 + k];
    }
    part[(size_t)blockIdx.x * 2 * channels + c] = a;
    part[((size_t)blockIdx.x * 2 + 1) * channels + c] = b;
  }
}

// Adds the blocks' sums: the affine gradients, and what the last pass subtracts,
// coef[0][c] = mean of dz and coef[1][c] = mean of dz * xhat * rstd.
__global__ void __launch_bounds__(kBnFinishThreads, 1)
bn_finish_sums_kernel(const float* __restrict__ part, int nparts, int channels, int64_t rows,
                      const float* __restrict__ rstd, float* __restrict__ dgamma, float* __restrict__ dbeta,
                      float* __restrict__ coef) {
  __shared__ double sm[kBnFinishThreads / 32][9];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 8 + (threadIdx.x & 7), row = threadIdx.x >> 3;
  float v1[kBnFinishLoads], v2[kBnFinishLoads];
#pragma unroll
  for (int j = 0; j < kBnFinishLoads; ++j) {
    const int b = row + j * kBnFinishRows;
    v1[j] = b < nparts ? part[(size_t)b * 2 * channels + c] : 0.f;
    v2[j] = b < nparts ? part[((size_t)b * 2 + 1) * channels + c] : 0.f;
  }
  double t1 = 0.0, t2 = 0.0;
#pragma unroll
  for (int j = 0; j < kBnFinishLoads; ++j) {
    t1 += v1[j];
    t2 += v2[j];
  }
  t1 = sumOfChannel(t1, sm);
  t2 = sumOfChannel(t2, sm);
  const int mine = blockIdx.x * 8 + w;
  if (lane == 0 && w < 8) {
    const double r = rstd[mine];
    dbeta[mine] = (float)t1;
    dgamma[mine] = (float)(t2 * r);
    coef[mine] = (float)(t1 / (double)rows);
    coef[channels + mine] = (float)(t2 * r * r / (double)rows);
  }
}

// dx = gamma * rstd * (dz - mean(dz) - xhat * mean(dz * xhat)); `dz` is dy itself
// with kBnNone, dy in front of the mask with kBnFromX, else already masked.
template <typename T, bool kFromX>
__global__ void __launch_bounds__(kBnThreads, 3)
bn_bwd_dx_kernel(const T* __restrict__ dz, const T* __restrict__ x, T* __restrict__ dx,
                 const float* __restrict__ mean, const float* __restrict__ rstd,
                 const float* __restrict__ gamma, const float* __restrict__ beta,
                 const float* __restrict__ coef, int64_t nvec, int groups) {
  constexpr int U = 2;
  const int group = threadIdx.x % groups;
  float mu[8], scale[8], shift[8], c1[8], c2[8];
  loadChannels(mean, group, mu);
  if constexpr (kFromX) loadChannels(beta, group, shift);
  loadChannels(coef, group, c1);
  loadChannels(coef + groups * 8, group, c2);
  {
    float g[8];
    loadChannels(rstd, group, scale);
    loadChannels(gamma, group, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) scale[k] *= g[k];
  }
  const int64_t stride = (int64_t)gridDim.x * kBnThreads;
  auto one = [&](const Raw8<T>& rd, const Raw8<T>& rx, int64_t at) {
    float d[8], v[8];
    rd.get(d);
    rx.get(v);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float e = v[k] - mu[k];
      if constexpr (kFromX) d[k] = fmaf(e, scale[k], shift[k]) <= 0.f ? 0.f : d[k];
      v[k] = scale[k] * (d[k] - c1[k] - e * c2[k]);
    }
    Raw8<T> out;
    out.set(v);
    out.store(dx + at * 8);
  };
  const int64_t first = (int64_t)blockIdx.x * kBnThreads + threadIdx.x;
  int64_t i = first < nvec ? first + (nvec - 1 - first) / stride * stride : -1;  // the thread's last vector
  for (; i - (U - 1) * stride >= 0; i -= U * stride) {
    Raw8<T> rd[U], rx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rd[u].load(dz + (i - u * stride) * 8);
      rx[u].load(x + (i - u * stride) * 8);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) one(rd[u], rx[u], i - u * stride);
  }
  for (; i >= 0; i -= stride) {
    Raw8<T> rd, rx;
    rd.load(dz + i * 8);
    rx.load(x + i * 8);
    one(rd, rx, i);
  }
}

unsigned streamBlocks(int64_t nvec, int per_sm, int sm_count) {
  const int64_t want = (nvec + kBnThreads - 1) / kBnThreads, cap = (int64_t)sm_count * per_sm;
  return (unsigned)(want < cap ? want : cap);
}

template <typename T>
cudaError_t forwardOf(const BatchNormShape& s, const void* x, const void* residual, void* y, bool relu,
                      const float* gamma, const float* beta, float* mean, float* rstd, float* running_mean,
                      float* running_var, int64_t* tracked, float momentum, float eps, float* part,
                      int sm_count, cudaStream_t stream) {
  const int groups = s.channels / 8;
  const int64_t nvec = s.rows * groups;
  const int nparts = batchNormParts(s, sm_count);
  const T* xt = static_cast<const T*>(x);
  const T* rt = static_cast<const T*>(residual);
  T* yt = static_cast<T*>(y);
  bn_stats_kernel<T><<<nparts, kBnThreads, 0, stream>>>(xt, nvec, groups, part);
  bn_finish_stats_kernel<<<s.channels / 8, kBnFinishThreads, 0, stream>>>(
      part, nparts, kBnThreads / groups, s.channels, s.rows, eps, momentum, mean, rstd, running_mean, running_var, tracked);
  const unsigned blocks = streamBlocks(nvec, 4, sm_count);
#define FR_BN_APPLY(R, A) \
  bn_apply_kernel<T, R, A><<<blocks, kBnThreads, 0, stream>>>(xt, rt, yt, mean, rstd, gamma, beta, nvec, groups)
  if (rt != nullptr) {
    if (relu) FR_BN_APPLY(true, true); else FR_BN_APPLY(false, true);
  } else {
    if (relu) FR_BN_APPLY(true, false); else FR_BN_APPLY(false, false);
  }
#undef FR_BN_APPLY
  return cudaGetLastError();
}

template <typename T>
cudaError_t backwardOf(const BatchNormShape& s, const void* dy, const void* dy2, const void* x, const void* y, void* dz, void* dx,
                       bool relu, const float* gamma, const float* beta, const float* mean, const float* rstd,
                       float* dgamma, float* dbeta, float* part, int sm_count, cudaStream_t stream) {
  const int groups = s.channels / 8;
  const int64_t nvec = s.rows * groups;
  const int nparts = batchNormParts(s, sm_count);
  const T* dyt = static_cast<const T*>(dy);
  const T* dy2t = static_cast<const T*>(dy2);
  const T* xt = static_cast<const T*>(x);
  const T* yt = static_cast<const T*>(y);
  T* dzt = static_cast<T*>(dz);
  T* dxt = static_cast<T*>(dx);
  float* coef = part + (size_t)nparts * 2 * s.channels;
#define FR_BN_SUMS(...)                                                                                       \
  bn_bwd_sums_kernel<T, __VA_ARGS__><<<nparts, kBnThreads, 0, stream>>>(dyt, dy2t, xt, yt, dzt, mean, rstd, gamma, \
                                                                        beta, nvec, groups, part)
  if (!relu) FR_BN_SUMS(kBnNone);
  else if (yt == nullptr) FR_BN_SUMS(kBnFromX);
  else if (dy2t == nullptr) FR_BN_SUMS(kBnFromY);
  else FR_BN_SUMS(kBnFromY, true);
#undef FR_BN_SUMS
  bn_finish_sums_kernel<<<s.channels / 8, kBnFinishThreads, 0, stream>>>(
      part, nparts, s.channels, s.rows, rstd, dgamma, dbeta, coef);
  const unsigned blocks = streamBlocks(nvec, 3, sm_count);
  if (relu && yt == nullptr)
    bn_bwd_dx_kernel<T, true><<<blocks, kBnThreads, 0, stream>>>(dyt, xt, dxt, mean, rstd, gamma, beta, coef, nvec, groups);
  else
    bn_bwd_dx_kernel<T, false><<<blocks, kBnThreads, 0, stream>>>(relu ? dzt : dyt, xt, dxt, mean, rstd, gamma, beta,
                                                                  coef, nvec, groups);
  return cudaGetLastError();
}

bool takes(const BatchNormShape& s) {
  return s.rows > 1 && s.channels >= 8 && s.channels <= 8 * kBnThreads && (s.channels & (s.channels - 1)) == 0;
}

}  // namespace

// One block per 32 rows of a thread, at least one block per SM and at most four:
// every block adds 8 bytes per channel that the small kernel has to read again.
int batchNormParts(const BatchNormShape& s, int sm_count) {
  const int64_t members = kBnThreads / (s.channels / 8);
  int64_t want = s.rows / (members * 32);
  if (want < sm_count) want = sm_count;
  if (want > (int64_t)sm_count * 4) want = (int64_t)sm_count * 4;
  const int64_t most = (s.rows + members - 1) / members;
  if (want > most) want = most;
  if (want > kBnMaxBlocks) want = kBnMaxBlocks;
  return (int)want;
}

int64_t batchNormScratchFloats(const BatchNormShape& s, int sm_count) {
  const int64_t nparts = batchNormParts(s, sm_count);
  return nparts * 2 * s.channels + 2 * s.channels;
}

cudaError_t launchBatchNormForward(const BatchNormShape& s, bool bf16, const void* x, const void* residual, void* y,
                                   bool relu, const float* gamma, const float* beta, float* mean, float* rstd,
                                   float* running_mean, float* running_var, int64_t* tracked, float momentum,
                                   float eps, float* scratch, int sm_count, cudaStream_t stream) {
  if (!takes(s)) return cudaErrorInvalidValue;
  const cudaError_t e =
      bf16 ? forwardOf<__nv_bfloat16>(s, x, residual, y, relu, gamma, beta, mean, rstd, running_mean, running_var,
                                      tracked, momentum, eps, scratch, sm_count, stream)
           : forwardOf<float>(s, x, residual, y, relu, gamma, beta, mean, rstd, running_mean, running_var, tracked,
                              momentum, eps, scratch, sm_count, stream);
  for (int i = 0; i < 3; ++i) noteLocalLaunch();
  return e;
}

cudaError_t launchBatchNormBackward(const BatchNormShape& s, bool bf16, const void* dy, const void* dy2, const void* x,
                                    const void* y, void* dz, void* dx, bool relu, const float* gamma, const float* beta,
                                    const float* mean, const float* rstd, float* dgamma, float* dbeta,
                                    float* scratch, int sm_count, cudaStream_t stream) {
  if (!takes(s) || (dy2 != nullptr && (y == nullptr || !relu))) return cudaErrorInvalidValue;
  const cudaError_t e =
      bf16 ? backwardOf<__nv_bfloat16>(s, dy, dy2, x, y, dz, dx, relu, gamma, beta, mean, rstd, dgamma, dbeta, scratch,
                                       sm_count, stream)
           : backwardOf<float>(s, dy, dy2, x, y, dz, dx, relu, gamma, beta, mean, rstd, dgamma, dbeta, scratch, sm_count,
                               stream);
  for (int i = 0; i < 3; ++i) noteLocalLaunch();
  return e;
}

}  // namespace fairring
