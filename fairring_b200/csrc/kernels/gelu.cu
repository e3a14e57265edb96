// What stands between the two GEMMs of a bf16 MLP (sm_100a): GELU, its backward,
// and the bias gradients of the linear layers, which are column sums over the
// gradient of their output.
//
// torch runs the GELU backward and the column sum of its result as two passes,
// and its column sum of a [rows, cols] bf16 matrix takes more than twice the time
// of reading it.  Here the GELU backward adds up the columns of what it writes,
// and a plain column sum serves the layers without an activation.  All three
// kernels are bound by HBM (or by L2, where the gradient was just written): 16-byte
// accesses, several rows in flight per thread.
//
// 8192 x 8192 bf16 (134 MB), tanh form: GELU 77 -> 49 us (5.5 TB/s); its backward and
// the bias gradient 97 + about 45 -> 79 + 4 us (5.1 TB/s; the erf form takes 109 us,
// bound by erff).  A plain column sum of the other layers of that block (6144 and
// 2048 wide): 28 us on average -> 12 + 4 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "local_kernels.h"
#include "vec8.cuh"

namespace fairring {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kGeluThreads = 256;

// tanh form: x * sigmoid(2u), u = sqrt(2/pi) (x + 0.044715 x^3); unlike 1 + tanh(u) it
// does not cancel for negative x.
constexpr float kTwoSqrt2OverPi = 1.5957691216057308f, kGeluCubic = 0.044715f;
__device__ __forceinline__ float sigmoidOf(float t) { return __fdividef(1.f, 1.f + __expf(-t)); }

template <bool kTanh>
__device__ __forceinline__ float gelu(float x) {
  if constexpr (kTanh) {
    return x * sigmoidOf(kTwoSqrt2OverPi * (x + kGeluCubic * x * x * x));
  } else {
    return x * 0.5f * (1.f + erff(x * 0.70710678118654752f));
  }
}

template <bool kTanh>
__device__ __forceinline__ float geluGrad(float x) {
  if constexpr (kTanh) {
    const float s = sigmoidOf(kTwoSqrt2OverPi * (x + kGeluCubic * x * x * x));
    return s + x * s * (1.f - s) * kTwoSqrt2OverPi * (1.f + 3.f * kGeluCubic * x * x);
  } else {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    return cdf + x * 0.3989422804014327f * __expf(-0.5f * x * x);
  }
}

template <bool kTanh>
__global__ void __launch_bounds__(kGeluThreads)
gelu_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, int64_t nvec) {
  constexpr int U = 4;
  const int64_t first = (int64_t)blockIdx.x * kGeluThreads * U + threadIdx.x;
  Raw8<bf16> r[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (first + u * kGeluThreads < nvec) r[u].load(x + (first + u * kGeluThreads) * 8);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (first + u * kGeluThreads < nvec) {
      float v[8];
      r[u].get(v);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = gelu<kTanh>(v[k]);
      r[u].set(v);
      r[u].store(y + (first + u * kGeluThreads) * 8);
    }
  }
}

enum ColumnSumOf { kOfInput, kOfTanhGelu, kOfErfGelu };
// Measured for 8192 x 8192 (tanh, erf) and the mean of 8192 x 6144 and 2048 (input), four blocks with
// half the loads in flight against three with all: 79 against 85 us, 112 against 109, 12.8 against 12.4.
template <ColumnSumOf kOf> constexpr int kColumnBlocksPerSm = kOf == kOfTanhGelu ? 4 : 3;

// partial[strip][c] = sum of column c over the strip's rows: of dy itself, or of
// dx = dy * gelu'(x), which is written out on the way.  A block is `wide` threads
// across the columns (8 each) and 256 / wide rows.
template <ColumnSumOf kOf>
__global__ void __launch_bounds__(kGeluThreads, kColumnBlocksPerSm<kOf>)
column_sum_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, bf16* __restrict__ dx,
                  float* __restrict__ partial, int64_t rows, int cols, int wide) {
  constexpr int U = kOf == kOfInput ? 8 : kOf == kOfTanhGelu ? 2 : 4;
  const int across = threadIdx.x % wide, down = threadIdx.x / wide, height = kGeluThreads / wide;
  const int c = (blockIdx.x * wide + across) * 8;
  const int64_t stride = (int64_t)gridDim.y * height;
  float acc[8] = {};
  if (c < cols) {
    for (int64_t r = (int64_t)blockIdx.y * height + down; r < rows; r += U * stride) {
      Raw8<bf16> d[U], h[kOf == kOfInput ? 1 : U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t row = r + u * stride;
        if (row < rows) {
          d[u].load(dy + row * cols + c);
          if constexpr (kOf != kOfInput) h[u].load(x + row * cols + c);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t row = r + u * stride;
        if (row < rows) {
          float v[8];
          d[u].get(v);
          if constexpr (kOf != kOfInput) {
            float e[8];
            h[u].get(e);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] *= geluGrad<kOf == kOfTanhGelu>(e[k]);
            d[u].set(v);
            d[u].store(dx + row * cols + c);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += v[k];
        }
      }
    }
  }
  if (height > 1) {
    __shared__ float sums[kGeluThreads * 9];
#pragma unroll
    for (int k = 0; k < 8; ++k) sums[threadIdx.x * 9 + k] = acc[k];
    __syncthreads();
    if (down != 0) return;
    for (int m = 1; m < height; ++m) {
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += sums[(m * wide + across) * 9 + k];
    }
  }
  if (c < cols) {
    Raw8<float> out;
    out.set(acc);
    out.store(partial + (size_t)blockIdx.y * cols + c);
  }
}

// Adds the strips, 32 columns per block, one strip per warp at a time.
template <typename T>
__global__ void __launch_bounds__(1024, 1)
column_sum_finish_kernel(const float* __restrict__ partial, int strips, int cols, T* __restrict__ out) {
  constexpr int W = 32, U = 8;
  __shared__ float acc[W][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < cols) {
    for (int b = w; b < strips; b += W * U) {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = b + u * W < strips ? partial[(size_t)(b + u * W) * cols + c] : 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u) s += v[u];
    }
  }
  acc[w][lane] = s;
  __syncthreads();
  s = acc[lane][w];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const int mine = blockIdx.x * 32 + w;
  if (lane == 0 && mine < cols) {
    if constexpr (sizeof(T) == 2)
      out[mine] = __float2bfloat16_rn(s);
    else
      out[mine] = s;
  }
}

struct ColumnGeometry {
  int wide = 1, tiles, strips;
  // As many blocks as are resident, but at least four rows for a thread: a strip is read
  // again by the finishing kernel.
  ColumnGeometry(int64_t rows, int cols, int sm_count, int per_sm) {
    while (wide < kGeluThreads && wide * 8 < cols) wide *= 2;
    tiles = (cols / 8 + wide - 1) / wide;
    const int64_t height = kGeluThreads / wide;
    int64_t n = ((int64_t)sm_count * per_sm + tiles - 1) / tiles;
    const int64_t most = (rows + 4 * height - 1) / (4 * height);
    strips = (int)(n < most ? n : most);
    if (strips < 1) strips = 1;
    if (strips > 65535) strips = 65535;
  }
};

bool takes(int cols) { return cols >= 8 && cols % 8 == 0; }

}  // namespace

cudaError_t launchGeluForward(const void* x, void* y, int64_t n, bool tanh_form, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  if (n % 8 != 0) return cudaErrorInvalidValue;
  const int64_t nvec = n / 8, blocks = (nvec + kGeluThreads * 4 - 1) / (kGeluThreads * 4);
  if (blocks > INT32_MAX) return cudaErrorInvalidValue;
  auto kernel = tanh_form ? gelu_fwd_kernel<true> : gelu_fwd_kernel<false>;
  kernel<<<(unsigned)blocks, kGeluThreads, 0, stream>>>(static_cast<const bf16*>(x), static_cast<bf16*>(y), nvec);
  noteLocalLaunch();
  return cudaGetLastError();
}

int columnSumStrips(int64_t rows, int cols, int sm_count) {
  return ColumnGeometry(rows, cols, sm_count, kColumnBlocksPerSm<kOfTanhGelu>).strips;  // the largest of the three
}

cudaError_t launchColumnSum(const void* dy, const void* gelu_x, bool tanh_form, void* dx, float* partial, void* out,
                            bool out_bf16, int64_t rows, int cols, int sm_count, cudaStream_t stream) {
  if (!takes(cols) || rows < 0) return cudaErrorInvalidValue;
  const ColumnGeometry g(rows, cols, sm_count,
                         gelu_x != nullptr && tanh_form ? kColumnBlocksPerSm<kOfTanhGelu> : kColumnBlocksPerSm<kOfInput>);
  auto kernel = gelu_x == nullptr ? column_sum_kernel<kOfInput>
                                  : (tanh_form ? column_sum_kernel<kOfTanhGelu> : column_sum_kernel<kOfErfGelu>);
  kernel<<<dim3(g.tiles, g.strips), kGeluThreads, 0, stream>>>(static_cast<const bf16*>(dy),
                                                               static_cast<const bf16*>(gelu_x),
                                                               static_cast<bf16*>(dx), partial, rows, cols, g.wide);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (out_bf16)
    column_sum_finish_kernel<bf16><<<(cols + 31) / 32, 1024, 0, stream>>>(partial, g.strips, cols, static_cast<bf16*>(out));
  else
    column_sum_finish_kernel<float><<<(cols + 31) / 32, 1024, 0, stream>>>(partial, g.strips, cols, static_cast<float*>(out));
  noteLocalLaunch();
  noteLocalLaunch();
  return cudaGetLastError();
}

}  // namespace fairring
