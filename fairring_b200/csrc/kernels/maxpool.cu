// Max pooling of channels-last activations (sm_100a).  torch keeps an int64 index
// per output, four times the bytes of the bf16 output itself, and its backward
// spends most of its time on them; here the position inside the window is one byte.
//
// Both kernels are bound by memory: a thread owns 8 channels of one pixel, neighbours
// in a warp the next channels and pixels, so loads are 16 bytes and what windows
// share comes from L1 and L2.  The backward gathers: an input pixel looks at the windows
// it lies in and takes the gradient of those that chose it, so nothing is zeroed first.
//
// 256 x 64 x 112 x 112 bf16, window 3, stride 2: forward 749 -> 200 us, backward 1731 ->
// 469 us against torch's kernels; both now spend their time on comparing and
// unpacking, 86 us would do for the bytes.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "local_kernels.h"
#include "vec8.cuh"

namespace fairring {
namespace {

constexpr int kPoolThreads = 256;

// Where vector i of a [images, height, width, groups] tensor lies.
struct Pixel {
  uint32_t group, w, h, image;
  __device__ __forceinline__ Pixel(uint32_t i, uint32_t groups, uint32_t width, uint32_t height) {
    const uint32_t p = i / groups, q = p / width;
    group = i - p * groups;
    w = p - q * width;
    image = q / height;
    h = q - image * height;
  }
};

// The first largest element of the window in row order, a NaN counting as largest.
template <typename T>
__global__ void __launch_bounds__(kPoolThreads)
max_pool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, uint2* __restrict__ chosen, PoolShape s,
                    uint32_t groups, uint32_t total) {
  const uint32_t i = blockIdx.x * kPoolThreads + threadIdx.x;
  if (i >= total) return;
  const Pixel o(i, groups, s.out_w, s.out_h);
  const int h0 = (int)o.h * s.stride - s.pad, w0 = (int)o.w * s.stride - s.pad;
  const T* image = x + (size_t)o.image * s.in_h * s.in_w * groups * 8 + o.group * 8;
  float best[8];
  uint32_t at[8];
  bool first = true;
  for (int kh = 0; kh < s.window; ++kh) {
    const int h = h0 + kh;
    if (h < 0 || h >= s.in_h) continue;
    for (int kw = 0; kw < s.window; ++kw) {
      const int w = w0 + kw;
      if (w < 0 || w >= s.in_w) continue;
      Raw8<T> r;
      r.load(image + ((size_t)h * s.in_w + w) * groups * 8);
      float v[8];
      r.get(v);
      const uint32_t k = kh * s.window + kw;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (first || v[c] > best[c] || v[c] != v[c]) {
          best[c] = v[c];
          at[c] = k;
        }
      }
      first = false;
    }
  }
  Raw8<T> out;
  out.set(best);
  out.store(y + (size_t)i * 8);
  chosen[i] = make_uint2(at[0] | at[1] << 8 | at[2] << 16 | at[3] << 24, at[4] | at[5] << 8 | at[6] << 16 | at[7] << 24);
}

template <typename T>
__global__ void __launch_bounds__(kPoolThreads)
max_pool_bwd_kernel(const T* __restrict__ dy, const uint2* __restrict__ chosen, T* __restrict__ dx, PoolShape s,
                    uint32_t groups, uint32_t total) {
  const uint32_t i = blockIdx.x * kPoolThreads + threadIdx.x;
  if (i >= total) return;
  const Pixel p(i, groups, s.in_w, s.in_h);
  const int h = (int)p.h + s.pad, w = (int)p.w + s.pad;
  // windows that cover the pixel
  const int oh0 = h < s.window ? 0 : (h - s.window) / s.stride + 1, oh1 = min(h / s.stride, s.out_h - 1);
  const int ow0 = w < s.window ? 0 : (w - s.window) / s.stride + 1, ow1 = min(w / s.stride, s.out_w - 1);
  const size_t image = (size_t)p.image * s.out_h * s.out_w;
  float sum[8] = {};
  for (int oh = oh0; oh <= oh1; ++oh) {
    for (int ow = ow0; ow <= ow1; ++ow) {
      const size_t o = (image + (size_t)oh * s.out_w + ow) * groups + p.group;
      const uint32_t k = (h - oh * s.stride) * s.window + (w - ow * s.stride);
      const uint2 at = chosen[o];
      Raw8<T> r;
      r.load(dy + o * 8);
      float v[8];
      r.get(v);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint32_t b = ((c < 4 ? at.x : at.y) >> (8 * (c & 3))) & 255u;
        sum[c] += b == k ? v[c] : 0.f;
      }
    }
  }
  Raw8<T> out;
  out.set(sum);
  out.store(dx + (size_t)i * 8);
}

// Every window has to hold an element, and a position has to fit a byte; 32-bit vector counts.
bool takes(const PoolShape& s) {
  const int64_t groups = s.channels / 8;
  return s.images > 0 && s.channels > 0 && s.channels % 8 == 0 && s.window >= 1 && s.window <= 16 && s.stride >= 1 &&
         s.pad >= 0 && 2 * s.pad <= s.window && s.in_h > 0 && s.in_w > 0 && s.out_h > 0 && s.out_w > 0 &&
         (int64_t)(s.out_h - 1) * s.stride - s.pad < s.in_h && (int64_t)(s.out_w - 1) * s.stride - s.pad < s.in_w &&
         (int64_t)s.images * s.in_h * s.in_w * groups < INT32_MAX && (int64_t)s.images * s.out_h * s.out_w * groups < INT32_MAX;
}

unsigned blocksFor(int64_t total) { return (unsigned)((total + kPoolThreads - 1) / kPoolThreads); }

}  // namespace

cudaError_t launchMaxPoolForward(const PoolShape& s, bool bf16, const void* x, void* y, void* chosen,
                                 cudaStream_t stream) {
  if (!takes(s)) return cudaErrorInvalidValue;
  const uint32_t groups = s.channels / 8, total = (uint32_t)s.images * s.out_h * s.out_w * groups;
  if (bf16)
    max_pool_fwd_kernel<__nv_bfloat16><<<blocksFor(total), kPoolThreads, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), static_cast<uint2*>(chosen), s, groups, total);
  else
    max_pool_fwd_kernel<float><<<blocksFor(total), kPoolThreads, 0, stream>>>(
        static_cast<const float*>(x), static_cast<float*>(y), static_cast<uint2*>(chosen), s, groups, total);
  noteLocalLaunch();
  return cudaGetLastError();
}

cudaError_t launchMaxPoolBackward(const PoolShape& s, bool bf16, const void* dy, const void* chosen, void* dx,
                                  cudaStream_t stream) {
  if (!takes(s)) return cudaErrorInvalidValue;
  const uint32_t groups = s.channels / 8, total = (uint32_t)s.images * s.in_h * s.in_w * groups;
  if (bf16)
    max_pool_bwd_kernel<__nv_bfloat16><<<blocksFor(total), kPoolThreads, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(dy), static_cast<const uint2*>(chosen), static_cast<__nv_bfloat16*>(dx), s, groups, total);
  else
    max_pool_bwd_kernel<float><<<blocksFor(total), kPoolThreads, 0, stream>>>(
        static_cast<const float*>(dy), static_cast<const uint2*>(chosen), static_cast<float*>(dx), s, groups, total);
  noteLocalLaunch();
  return cudaGetLastError();
}

}  // namespace fairring
