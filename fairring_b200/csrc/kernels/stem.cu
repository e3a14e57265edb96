// The input of a 7 x 7, stride 2 convolution over 3 channels, folded (sm_100a).
//
// Three channels give a tensor-core convolution rows of 6 bytes. Over the 2 x 2
// pixel blocks of the image, 12 channels and 4 zeros, the same convolution is a 4 x 4
// one of stride 1 over 16 channels, 32 bytes a pixel: block row p holds the rows
// 2 (p - 2) and 2 (p - 2) + 1, output row r reads the blocks r to r + 3, and the first
// row and column of the 8 x 8 kernel that this makes are zero (a pixel that is not
// finite makes the outputs that these meet NaN as well). The fold also rounds to
// bf16 and pads, so it replaces the cast in front of the convolution. Bound by HBM.
//
// 256 images of 224 x 224, 64 output channels: the convolution takes 0.53 ms folded and
// 1.60 ms as it is. Its weight gradient takes 1.56 ms folded and 0.91 ms as it is, so
// that one stays with the image.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "local_kernels.h"
#include "vec8.cuh"

namespace fairring {
namespace {

__device__ __forceinline__ float pixelOf(float v) { return v; }
__device__ __forceinline__ float pixelOf(__nv_bfloat16 v) { return __bfloat162float(v); }

// One thread per block of the folded image.
template <typename T>
__global__ void __launch_bounds__(256)
stem_fold_kernel(const T* __restrict__ image, __nv_bfloat16* __restrict__ out, int height, int width, uint32_t rows,
                 uint32_t cols, uint32_t total) {
  const uint32_t i = blockIdx.x * 256u + threadIdx.x;
  if (i >= total) return;
  const uint32_t t = i / cols, q = i - t * cols, n = t / rows, p = t - n * rows;
  float v[16] = {};
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const int h = 2 * ((int)p - 2) + b;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int w = 2 * ((int)q - 2) + a;
      if (h >= 0 && h < height && w >= 0 && w < width) {
        const T* src = image + (((size_t)n * height + h) * width + w) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[(b * 2 + a) * 3 + c] = pixelOf(src[c]);
      }
    }
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = v[half * 8 + k];
    Raw8<__nv_bfloat16> r;
    r.set(e);
    r.store(out + (size_t)i * 16 + half * 8);
  }
}

}  // namespace

cudaError_t launchStemFold(const void* image, bool bf16, void* out, int images, int height, int width, int rows,
                           int cols, cudaStream_t stream) {
  const int64_t total = (int64_t)images * rows * cols;
  if (total <= 0) return cudaSuccess;
  if (total > INT32_MAX) return cudaErrorInvalidValue;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (bf16)
    stem_fold_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(image),
                                                                static_cast<__nv_bfloat16*>(out), height, width, rows,
                                                                cols, (uint32_t)total);
  else
    stem_fold_kernel<float><<<blocks, 256, 0, stream>>>(static_cast<const float*>(image),
                                                        static_cast<__nv_bfloat16*>(out), height, width, rows, cols,
                                                        (uint32_t)total);
  noteLocalLaunch();
  return cudaGetLastError();
}

}  // namespace fairring
