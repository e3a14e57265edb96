// Softmax cross-entropy over a [rows, vocab] logits matrix (sm_100a) for the
// language-model workloads.  torch's path under bf16 autocast widens the bf16
// logits to fp32 (a pass), runs log_softmax (a pass each way), nll_loss, and
// narrows the fp32 gradient back to bf16 (another pass): more than ten bytes of
// HBM traffic per logit.  Here the forward reads every logit once and keeps the
// logarithm of a row's sum as two floats; the backward recomputes the softmax from the
// logits and those and writes the gradient in the logits' own dtype: six bytes per bf16
// logit in all, which is what bounds both kernels.
//
// Rows of any length: a row is the elements up to its first 16-byte boundary, 16-byte
// vectors, and what is left behind them.  All vectors of a batch are loaded
// before the first is used.
//
// 1229 x 50265 bf16, an odd vocabulary: torch's kernels and casts take 620 us in both
// directions, these 82 us.  8192 x 51200 bf16: forward 189 us (4.4 TB/s; exp() and the
// conversions around it keep the issue slots about half busy; 212 us with 512 threads
// that use a batch before they load the next), backward 276 us (6.1 TB/s; 289 us with
// a block per row instead of per batch), the mean 4 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cassert>
#include <cstdint>

#include "local_kernels.h"

namespace fairring {
namespace {

constexpr int kCeBatch = 4;  // 16-byte vectors in flight per thread

__device__ __forceinline__ float toFloat(float v) { return v; }
__device__ __forceinline__ float toFloat(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void fromFloat(float* p, float v) { *p = v; }
__device__ __forceinline__ void fromFloat(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// exp() of a difference of logits.  The fast form's relative error grows with the argument (2 + 1.17 |x|
// units in the last place of fp32): far below bf16's rounding, but not below that of fp32 results.
template <typename T> __device__ __forceinline__ float expOf(float v);
template <> __device__ __forceinline__ float expOf<float>(float v) { return expf(v); }
template <> __device__ __forceinline__ float expOf<__nv_bfloat16>(float v) { return __expf(v); }

template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int kElems = 4;
  static constexpr uint32_t kMinusInf = 0xff800000u;
  static __device__ __forceinline__ void get(const uint4& r, float (&v)[4]) {
    v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
  }
  static __device__ __forceinline__ float max(const uint4& r) {
    float v[4];
    get(r, v);
    return fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
  }
  static __device__ __forceinline__ uint4 set(const float (&v)[4]) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  }
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int kElems = 8;
  static constexpr uint32_t kMinusInf = 0xff80ff80u;
  static __device__ __forceinline__ void get(const uint4& r, float (&v)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ float max(const uint4& r) {  // packed: half the comparisons
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
    const float2 m = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
    return fmaxf(m.x, m.y);
  }
  static __device__ __forceinline__ uint4 set(const float (&v)[8]) {
    uint4 r;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    return r;
  }
};

// A row: `head` elements, `nvec` aligned 16-byte vectors, `tail` elements.
template <typename T> struct RowParts {
  int head, nvec, tail;
  __device__ __forceinline__ RowParts(const T* row, int vocab) {
    constexpr int E = Vec16<T>::kElems;
    const int off = (int)(reinterpret_cast<uintptr_t>(row) & 15u) / (int)sizeof(T);
    head = min(vocab, (E - off) % E);
    nvec = (vocab - head) / E;
    tail = vocab - head - nvec * E;
  }
};

// A running maximum and the sum of exp(value - maximum) below it.
template <typename T> struct SoftSum {
  float m = -INFINITY, s = 0.f;
  // What exp() is taken relative to: never -inf, whose difference from itself is NaN.
  static __device__ __forceinline__ float reference(float m) { return m == -INFINITY ? 0.f : m; }
  __device__ __forceinline__ void add(float v) {
    const float m_new = fmaxf(m, v), ref = reference(m_new);
    s = s * expOf<T>(m - ref) + expOf<T>(v - ref);
    m = m_new;
  }
};

template <int kThreads>
__device__ __forceinline__ float blockReduce(float v, bool is_max, float* scratch) {
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, other) : v + other;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = scratch[0];
#pragma unroll
  for (int i = 1; i < kThreads / 32; ++i) r = is_max ? fmaxf(r, scratch[i]) : r + scratch[i];
  return r;
}

// loss[r] = logsumexp(row r) - row r[target]; kept for the backward: logsumexp in lse[r] and what
// its rounding cut off in lse[kept + r].  At a maximum of 20 that is up to 1e-6 of every probability
// of the row, several times fp32's own error.
// A negative target marks a row that does not count: loss 0, as for a target past the
// vocabulary.  With `classes` > 0 a target that is neither below it nor -100 ends the program, as it
// does in torch's loss.  One block per row, one sweep over it: a thread
// rescales its sum once per batch of vectors when its maximum grew, and the next
// batch is on its way while this one is used.
template <typename T, int kThreads>
__global__ void __launch_bounds__(kThreads, 1280 / kThreads)
cross_entropy_fwd_kernel(const T* __restrict__ logits, const int64_t* __restrict__ targets,
                         float* __restrict__ loss, float* __restrict__ lse, int64_t kept, int vocab, int classes) {
  constexpr int E = Vec16<T>::kElems, U = kCeBatch;
  __shared__ float scratch[kThreads / 32];
  const int64_t r = blockIdx.x;
  const T* row = logits + r * vocab;
  const RowParts<T> parts(row, vocab);
  const uint4* vecs = reinterpret_cast<const uint4*>(row + parts.head);
  SoftSum<T> a;
  uint4 raw[U];
  auto fetch = [&](int i) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      constexpr uint32_t w = Vec16<T>::kMinusInf;
      raw[u] = i + u * kThreads < parts.nvec ? vecs[i + u * kThreads] : make_uint4(w, w, w, w);
    }
  };
  int i = threadIdx.x;
  fetch(i);
  while (i < parts.nvec) {
    uint4 now[U];
#pragma unroll
    for (int u = 0; u < U; ++u) now[u] = raw[u];
    i += U * kThreads;
    fetch(i);
    float top = a.m;
#pragma unroll
    for (int u = 0; u < U; ++u) top = fmaxf(top, Vec16<T>::max(now[u]));
    const float ref = SoftSum<T>::reference(top);
    float s[2] = {};
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float v[E];
      Vec16<T>::get(now[u], v);
#pragma unroll
      for (int k = 0; k < E; ++k) s[k & 1] += expOf<T>(v[k] - ref);
    }
    a.s = a.s * expOf<T>(a.m - ref) + (s[0] + s[1]);
    a.m = top;
  }
  if ((int)threadIdx.x < parts.head) a.add(toFloat(row[threadIdx.x]));
  if ((int)threadIdx.x < parts.tail) a.add(toFloat(row[vocab - parts.tail + threadIdx.x]));
  const float m = blockReduce<kThreads>(a.m, true, scratch);
  const float s = blockReduce<kThreads>(a.s * expOf<T>(a.m - SoftSum<T>::reference(m)), false, scratch);
  if (threadIdx.x == 0) {
    const float ls = logf(s), l = m + ls, part = l - m;
    lse[r] = l;
    lse[kept + r] = (m - (l - part)) + (ls - part);  // m + ls - l, exactly
    const int64_t t = targets[r];
    const bool counts = t >= 0 && t < vocab;
    assert((classes == 0 || t == -100 || (t >= 0 && t < classes)) && "target outside the vocabulary");
    loss[r] = counts ? (m - toFloat(row[t])) + ls : 0.f;
  }
}

// mean = sum of the rows' losses / how many rows count, count = that number
// (at least `least`).  One block: the launch bounds it, and five small kernels
// (compare, count, clamp, sum, divide) cost 17 us in its place.
__global__ void __launch_bounds__(1024)
cross_entropy_mean_kernel(const float* __restrict__ loss, const int64_t* __restrict__ targets, int64_t rows,
                          float least, float* __restrict__ mean, float* __restrict__ count) {
  __shared__ float scratch[32];
  float s = 0.f, n = 0.f;  // the count is exact up to 2^24 rows, beyond that as good as the sum of the losses
  for (int64_t r = threadIdx.x; r < rows; r += 1024) {
    s += loss[r];
    n += targets[r] >= 0 ? 1.f : 0.f;
  }
  s = blockReduce<1024>(s, false, scratch);
  n = blockReduce<1024>(n, false, scratch);
  if (threadIdx.x == 0) {
    n = fmaxf(n, least);
    *mean = s / n;
    *count = n;
  }
}

// grad[r][j] <- (softmax(row r)[j] - [j == target]) * (*upstream) / (*count) * scale;
// grad may be the logits.  A block does one batch of vectors of one row, so that all
// blocks are alike whatever the vocabulary.
template <typename T, int kThreads>
__global__ void __launch_bounds__(kThreads)
cross_entropy_bwd_kernel(const T* logits, T* grad, const int64_t* __restrict__ targets,
                         const float* __restrict__ lse, const float* __restrict__ upstream,
                         const float* __restrict__ count, float scale, int64_t kept, int64_t pieces_total, int pieces, int vocab) {
  constexpr int E = Vec16<T>::kElems, U = kCeBatch;
  const float g = (count != nullptr ? *upstream / *count : *upstream) * scale;
  for (int64_t w = blockIdx.x; w < pieces_total; w += gridDim.x) {
    const int64_t r = w / pieces;
    const int piece = (int)(w - r * pieces);
    const T* row = logits + r * vocab;
    T* out = grad + r * vocab;
    const RowParts<T> parts(row, vocab);
    const int first = piece * U * kThreads + threadIdx.x;
    const uint4* vecs = reinterpret_cast<const uint4*>(row + parts.head);
    uint4* vout = reinterpret_cast<uint4*>(out + parts.head);
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (first + u * kThreads < parts.nvec) raw[u] = vecs[first + u * kThreads];
    const int64_t t64 = targets[r];
    const bool counts = t64 >= 0 && t64 < vocab;
    const int t = counts ? (int)t64 : -1;
    const float l = lse[r], cut = sizeof(T) == 4 ? lse[kept + r] : 0.f;  // far below bf16's rounding
    auto one = [&](float v, int j) { return counts ? (expOf<T>(sizeof(T) == 4 ? (v - l) - cut : v - l) - (j == t ? 1.f : 0.f)) * g : 0.f; };
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = first + u * kThreads;
      if (i < parts.nvec) {
        float v[E];
        Vec16<T>::get(raw[u], v);
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] = one(v[k], parts.head + i * E + k);
        vout[i] = Vec16<T>::set(v);
      }
    }
    if (piece == 0) {
      const int h = threadIdx.x;
      if (h < parts.head) fromFloat(out + h, one(toFloat(row[h]), h));
      const int e = vocab - parts.tail + (int)threadIdx.x;
      if ((int)threadIdx.x < parts.tail) fromFloat(out + e, one(toFloat(row[e]), e));
    }
  }
}

constexpr int kCeFwdWide = 256, kCeFwdNarrow = 128, kCeBwdThreads = 256;

template <typename T>
void forwardOf(const void* logits, const int64_t* targets, float* loss, float* lse, int64_t rows, int vocab,
               int classes, cudaStream_t stream) {
  // A row that one batch of 256 threads would not fill takes 128.
  for (int64_t done = 0; done < rows; done += 1 << 30) {
    const unsigned n = (unsigned)(rows - done < (1 << 30) ? rows - done : (1 << 30));
    const T* at = static_cast<const T*>(logits) + done * vocab;
    if (vocab >= kCeFwdWide * kCeBatch * Vec16<T>::kElems)
      cross_entropy_fwd_kernel<T, kCeFwdWide><<<n, kCeFwdWide, 0, stream>>>(at, targets + done, loss + done, lse + done,
                                                                           rows, vocab, classes);
    else
      cross_entropy_fwd_kernel<T, kCeFwdNarrow><<<n, kCeFwdNarrow, 0, stream>>>(at, targets + done, loss + done,
                                                                               lse + done, rows, vocab, classes);
    noteLocalLaunch();
  }
}

template <typename T>
void backwardOf(const void* logits, void* grad, const int64_t* targets, const float* lse, const float* upstream,
                const float* count, float scale, int64_t rows, int vocab, cudaStream_t stream) {
  constexpr int per_piece = kCeBwdThreads * kCeBatch * Vec16<T>::kElems;
  const int pieces = (vocab + per_piece - 1) / per_piece;
  const int64_t total = rows * pieces;
  const unsigned blocks = (unsigned)(total < (1 << 30) ? total : (1 << 30));
  cross_entropy_bwd_kernel<T, kCeBwdThreads><<<blocks, kCeBwdThreads, 0, stream>>>(
      static_cast<const T*>(logits), static_cast<T*>(grad), targets, lse, upstream, count, scale, rows, total, pieces, vocab);
  noteLocalLaunch();
}

}  // namespace

cudaError_t launchCrossEntropyForward(const void* logits, bool bf16, const int64_t* targets, float* loss,
                                      float* lse, int64_t rows, int vocab, int classes, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  if (vocab <= 0) return cudaErrorInvalidValue;
  if (bf16)
    forwardOf<__nv_bfloat16>(logits, targets, loss, lse, rows, vocab, classes, stream);
  else
    forwardOf<float>(logits, targets, loss, lse, rows, vocab, classes, stream);
  return cudaGetLastError();
}

cudaError_t launchCrossEntropyMean(const float* loss, const int64_t* targets, int64_t rows, float least,
                                   float* mean, float* count, cudaStream_t stream) {
  cross_entropy_mean_kernel<<<1, 1024, 0, stream>>>(loss, targets, rows, least, mean, count);
  noteLocalLaunch();
  return cudaGetLastError();
}

cudaError_t launchCrossEntropyBackward(const void* logits, void* grad, bool bf16, const int64_t* targets,
                                       const float* lse, const float* upstream, const float* count, float scale,
                                       int64_t rows, int vocab, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  if (vocab <= 0) return cudaErrorInvalidValue;
  // A vector of the logits becomes a vector of the gradient.
  if ((reinterpret_cast<uintptr_t>(logits) ^ reinterpret_cast<uintptr_t>(grad)) & 15u) return cudaErrorMisalignedAddress;
  if (bf16)
    backwardOf<__nv_bfloat16>(logits, grad, targets, lse, upstream, count, scale, rows, vocab, stream);
  else
    backwardOf<float>(logits, grad, targets, lse, upstream, count, scale, rows, vocab, stream);
  return cudaGetLastError();
}

}  // namespace fairring
