// The input embedding of the language models, whose table is also the output
// projection (sm_100a): x = table[token] + position, and the gradient of the table
// from both of its uses.
//
// torch makes a dense gradient of the table for the lookup (fill, sort, segment sums),
// widens the projection's bf16 gradient to another, and adds the two: more than 2 GB
// for a 51200 x 2048 table.  Here the projection's gradient is widened once and the
// rows of the lookup are added into it where they belong, those of one token by one
// block in a fixed order; other blocks of the same launch sum the positions' gradient.
// Bound by HBM, by the widening above all: of a 51200 x 2048 table 1.1 ms -> 0.2 ms, for
// 8192 tokens 30 us forward and 50 us backward besides.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cassert>
#include <cstdint>

#include "local_kernels.h"

namespace fairring {
namespace {

constexpr int kEmbThreads = 256;

__device__ __forceinline__ float4 operator+(const float4& a, const float4& b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// One block per token and 4 x 256 columns.  A token outside the table ends the program, as it does
// in torch's embedding; nothing is read for it.
__global__ void __launch_bounds__(kEmbThreads)
embed_fwd_kernel(const int64_t* __restrict__ tokens, const float4* __restrict__ table, const float4* __restrict__ pos,
                 float4* __restrict__ x, int seq, int64_t vocab, int d4) {
  const int c = blockIdx.y * kEmbThreads + threadIdx.x;
  if (c >= d4) return;
  const int64_t r = blockIdx.x, t = tokens[r];
  const bool inside = t >= 0 && t < vocab;
  assert(inside && "token outside the table");
  if (inside) x[r * d4 + c] = table[t * d4 + c] + pos[(r % seq) * d4 + c];
}

// One block per position and 4 x 256 columns: the sum over the sequences.
__device__ __forceinline__ void sumPositions(const float4* __restrict__ dx, float4* __restrict__ dpos, int64_t s, int chunk,
                                             int batch, int seq, int d4) {
  const int c = chunk * kEmbThreads + threadIdx.x;
  if (c >= d4) return;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int b = 0; b < batch; ++b) sum = sum + dx[((int64_t)b * seq + s) * d4 + c];
  dpos[s * d4 + c] = sum;
}

// The rows of the tokens that are `bucket` modulo `buckets`, 4 x 64 columns, added to the table's
// gradient.  All of a token's rows meet in one block, so they are added without atomics and in an order that
// depends on the tokens alone.  The block looks through all tokens, kTile at a time, and lists
// its own in their order.  From a long list it takes out the frequent tokens, whose rows all warps share; of
// the rest, where looking for equal tokens pair by pair is cheap, a warp takes a token at a time.
//
// With the positions' sums, rows of 2048: 8192 tokens of 51200 50 us (by atomics, in no fixed order, 33 us), with 15 %
// of them one and the same 80 us (39), with all of them 272 us (83); a block's latency bounds the latter two.
constexpr int kTile = 8 * kEmbThreads;  // tokens per round, 8 to a thread
constexpr int kWarps = kEmbThreads / 32;
constexpr int kLong = 64;     // entries
constexpr int kFrequent = 4;  // of 32 entries looked at
constexpr int kWide = 2;      // float4 columns of a thread, 32 apart

struct TokenLists {
  alignas(16) uint32_t key[kTile + 4];  // token / buckets; no token's behind the last entry
  uint16_t at[kTile];                   // place within the round
  uint16_t next[kTile];                 // the next entry of the same token, or the list's length
  uint16_t count[kTile];                // entries of the token, 0 where this is not its first
  uint16_t rows[kTile];                 // places of the frequent token at hand
  float4 part[kWide][kWarps][32];
  int total[kWarps];
};

// Where a thread's `found` entries go, behind those of the threads before it, and the number of all.
__device__ __forceinline__ int2 placeOf(int found, TokenLists& l) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int upto = found;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += up;
  }
  __syncthreads();  // `total` may still be read, and so may the lists that are about to be written
  if (lane == 31) l.total[w] = upto;
  __syncthreads();
  int before = upto - found, all = 0;
#pragma unroll
  for (int v = 0; v < kWarps; ++v) {
    if (v < w) before += l.total[v];
    all += l.total[v];
  }
  return make_int2(before, all);
}

// The rows in l.rows, shared among the warps, added to a row of the table.
__device__ __forceinline__ void sumFrequent(const float4* __restrict__ row, float4* out, int c, int d4, int count,
                                            TokenLists& l) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int U = 4;
  float4 sum[kWide];
#pragma unroll
  for (int k = 0; k < kWide; ++k) sum[k] = zero;
  for (int e = w; e < count; e += U * kWarps) {
    float4 g[U][kWide];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int at = e + u * kWarps;
#pragma unroll
      for (int k = 0; k < kWide; ++k)
        g[u][k] = at < count && c + k * 32 < d4 ? row[(int64_t)l.rows[at] * d4 + k * 32] : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int k = 0; k < kWide; ++k) sum[k] = sum[k] + g[u][k];
    }
  }
#pragma unroll
  for (int k = 0; k < kWide; ++k) l.part[k][w][lane] = sum[k];
  __syncthreads();
  if (w < kWide && c + w * 32 < d4) {
    float4 all = l.part[w][0][lane];
#pragma unroll
    for (int v = 1; v < kWarps; ++v) all = all + l.part[w][v][lane];
    out[w * 32] = out[w * 32] + all;
  }
  __syncthreads();
}

__device__ __forceinline__ void sumTokens(const float4* __restrict__ dx, const int64_t* __restrict__ tokens,
                                          float4* dtable, uint32_t bucket, uint32_t buckets, int chunk, int64_t n,
                                          int64_t vocab, int d4, TokenLists& l) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = chunk * 32 * kWide + lane;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto tableRow = [&](uint32_t key) { return dtable + ((int64_t)key * buckets + bucket) * d4 + c; };
  for (int64_t base = 0; base < n; base += kTile) {
    uint32_t hits = 0;
    uint32_t key[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t i = base + threadIdx.x * 8 + k, t = i < n ? tokens[i] : -1;
      key[k] = (uint32_t)t / buckets;
      if (t >= 0 && t < vocab && (uint32_t)t - key[k] * buckets == bucket) hits |= 1u << k;
    }
    const int2 place = placeOf(__popc(hits), l);
    int m = place.y, slot = place.x;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (hits >> k & 1u) {
        l.key[slot] = key[k];
        l.at[slot++] = (uint16_t)(threadIdx.x * 8 + k);
      }
    }
    __syncthreads();
    const float4* row = dx + base * d4 + c;
    while (m > kLong) {
      const uint32_t sample = l.key[(2 * lane + 1) * m / 64];
      const unsigned best = __reduce_max_sync(0xffffffffu, __popc(__match_any_sync(0xffffffffu, sample)) * 32u + lane);
      if (best < kFrequent * 32u) break;
      const uint32_t own = __shfl_sync(0xffffffffu, sample, best & 31u);  // the same in all warps
      uint32_t mine = 0, other = 0, keys[8];
      uint16_t ats[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int i = threadIdx.x * 8 + k;
        if (i < m) {
          keys[k] = l.key[i];
          ats[k] = l.at[i];
          (keys[k] == own ? mine : other) |= 1u << k;
        }
      }
      const int2 to = placeOf(__popc(mine), l);
      int in = to.x, out = threadIdx.x * 8 - to.x;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (mine >> k & 1u) l.rows[in++] = ats[k];
        if (other >> k & 1u) {
          l.key[out] = keys[k];
          l.at[out++] = ats[k];
        }
      }
      __syncthreads();
      sumFrequent(row, tableRow(own), c, d4, to.y, l);
      m -= to.y;
    }
    if (threadIdx.x < 4) l.key[m + threadIdx.x] = ~0u;
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += kEmbThreads) {
      const uint32_t own = l.key[i];
      int before = 0, count = 0, next = m;
      for (int j = 0; j < m; j += 4) {
        const uint4 k = *reinterpret_cast<const uint4*>(l.key + j);
        const uint32_t there[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool hit = there[u] == own;
          count += hit;
          before += hit && j + u < i;
          if (hit && j + u > i) next = min(next, j + u);
        }
      }
      l.next[i] = (uint16_t)next;
      l.count[i] = (uint16_t)(before == 0 ? count : 0);
    }
    __syncthreads();
    for (int i = w; i < m; i += kWarps) {
      if (l.count[i] == 0) continue;
      float4* out = tableRow(l.key[i]);
      float4 was[kWide], sum[kWide];
#pragma unroll
      for (int k = 0; k < kWide; ++k) {
        was[k] = c + k * 32 < d4 ? out[k * 32] : zero;
        sum[k] = zero;
      }
      for (int e = i; e < m;) {
        float4 g[2][kWide];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
          for (int k = 0; k < kWide; ++k)
            g[u][k] = e < m && c + k * 32 < d4 ? row[(int64_t)l.at[e] * d4 + k * 32] : zero;
          if (e < m) e = l.next[e];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
          for (int k = 0; k < kWide; ++k) sum[k] = sum[k] + g[u][k];
        }
      }
#pragma unroll
      for (int k = 0; k < kWide; ++k)
        if (c + k * 32 < d4) out[k * 32] = was[k] + sum[k];
    }
    __syncthreads();  // the lists are used up; and a table row may go to another warp in the next round
  }
}

// The first `buckets` x `chunks` blocks do the tokens, the others the positions.
__global__ void __launch_bounds__(kEmbThreads, 4)
embed_bwd_kernel(const float4* __restrict__ dx, const int64_t* __restrict__ tokens, float4* dtable,
                 float4* __restrict__ dpos, int batch, int seq, int64_t vocab, int d4, uint32_t buckets, uint32_t chunks) {
  __shared__ TokenLists lists;
  const uint32_t token_blocks = buckets * chunks;
  if (blockIdx.x < token_blocks) {
    const uint32_t bucket = blockIdx.x / chunks;
    sumTokens(dx, tokens, dtable, bucket, buckets, (int)(blockIdx.x - bucket * chunks), (int64_t)batch * seq, vocab, d4,
              lists);
  } else {
    const uint32_t p = blockIdx.x - token_blocks;
    const uint32_t s = p % (uint32_t)seq;
    sumPositions(dx, dpos, s, (int)(p / (uint32_t)seq), batch, seq, d4);
  }
}

}  // namespace

cudaError_t launchEmbedForward(const int64_t* tokens, const float* table, const float* pos, float* x, int batch, int seq,
                               int64_t vocab, int d, cudaStream_t stream) {
  const int64_t rows = (int64_t)batch * seq;
  if (rows <= 0) return cudaSuccess;
  if (d <= 0 || d % 4 != 0 || rows > INT32_MAX) return cudaErrorInvalidValue;
  const int d4 = d / 4;
  const dim3 grid((unsigned)rows, (d4 + kEmbThreads - 1) / kEmbThreads);
  embed_fwd_kernel<<<grid, kEmbThreads, 0, stream>>>(tokens, reinterpret_cast<const float4*>(table),
                                                     reinterpret_cast<const float4*>(pos),
                                                     reinterpret_cast<float4*>(x), seq, vocab, d4);
  noteLocalLaunch();
  return cudaGetLastError();
}

cudaError_t launchEmbedBackward(const float* dx, const int64_t* tokens, float* dtable, float* dpos, int batch, int seq,
                                int64_t vocab, int d, int sm_count, cudaStream_t stream) {
  const int64_t n = (int64_t)batch * seq;
  if (n <= 0) return cudaSuccess;
  if (d <= 0 || d % 4 != 0 || vocab > UINT32_MAX) return cudaErrorInvalidValue;
  const int d4 = d / 4;
  const int64_t chunks = (d4 + 32 * kWide - 1) / (32 * kWide), position_blocks = (int64_t)seq * ((d4 + kEmbThreads - 1) / kEmbThreads);
  // As many token blocks as are resident, each of which looks through all tokens, but at least 8 tokens for one.
  int64_t buckets = (int64_t)sm_count * 4 / chunks;
  if (buckets > (n + 7) / 8) buckets = (n + 7) / 8;
  if (buckets < 1) buckets = 1;
  if (buckets * chunks + position_blocks > INT32_MAX) return cudaErrorInvalidValue;
  embed_bwd_kernel<<<(unsigned)(buckets * chunks + position_blocks), kEmbThreads, 0, stream>>>(
      reinterpret_cast<const float4*>(dx), tokens, reinterpret_cast<float4*>(dtable), reinterpret_cast<float4*>(dpos),
      batch, seq, vocab, d4, (uint32_t)buckets, (uint32_t)chunks);
  noteLocalLaunch();
  return cudaGetLastError();
}

}  // namespace fairring
