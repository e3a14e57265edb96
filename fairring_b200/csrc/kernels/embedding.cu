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
// 8192 tokens 30 us forward besides.
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

// The rows of the tokens that are `bucket` modulo `buckets`, 4 x 32 columns, added to the table's
// gradient.  All of a token's rows meet in one block, so they are added without atomics and in an order that
// depends on the tokens alone.  The block looks through all tokens, kTile at a time, and lists
// its own in their order; then a warp takes a token and walks through its rows, except that
// the rows of a frequent one are shared out among all warps.
constexpr int kTile = 8 * kEmbThreads;  // tokens per round, 8 to a thread
constexpr int kWarps = kEmbThreads / 32;
constexpr int kFrequent = 32;  // occurrences within a round

struct TokenLists {
  uint32_t key[kTile];    // token / buckets
  uint16_t at[kTile];     // place within the round
  uint16_t rank[kTile];   // how many entries of the same token come before
  uint16_t next[kTile];   // the one behind, or the list's length
  uint16_t count[kTile];  // all of them, where rank is 0
  uint16_t rows[kTile];   // of the frequent token at hand: its places by rank
  float4 part[kWarps][32];
  int total[kWarps];
};

__device__ __forceinline__ void sumTokens(const float4* __restrict__ dx, const int64_t* __restrict__ tokens,
                                          float4* dtable, uint32_t bucket, uint32_t buckets, int chunk, int64_t n,
                                          int64_t vocab, int d4, TokenLists& l) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = chunk * 32 + lane;
  const bool mine = c < d4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  int64_t t[8];
  auto fetch = [&](int64_t base) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t i = base + threadIdx.x * 8 + k;
      t[k] = i < n ? tokens[i] : -1;
    }
  };
  fetch(0);
  for (int64_t base = 0; base < n; base += kTile) {
    uint32_t hits = 0;
    uint32_t key[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      key[k] = (uint32_t)t[k] / buckets;
      if (t[k] >= 0 && t[k] < vocab && (uint32_t)t[k] - key[k] * buckets == bucket) hits |= 1u << k;
    }
    if (base + kTile < n) fetch(base + kTile);
    // where this thread's entries go: behind those of the threads before it
    const int found = __popc(hits);
    int before = found;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += up;
    }
    if (lane == 31) l.total[w] = before;
    __syncthreads();
    int m = 0, slot = before - found;
#pragma unroll
    for (int v = 0; v < kWarps; ++v) {
      if (v < w) slot += l.total[v];
      m += l.total[v];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (hits >> k & 1u) {
        l.key[slot] = key[k];
        l.at[slot++] = (uint16_t)(threadIdx.x * 8 + k);
      }
    }
    __syncthreads();
    bool frequent = false;
    for (int i = threadIdx.x; i < m; i += kEmbThreads) {
      const uint32_t own = l.key[i];
      int rank = 0, count = 0, next = m;
      for (int j = 0; j < m; ++j) {
        if (l.key[j] == own) {
          ++count;
          if (j < i) ++rank;
          if (j > i && next == m) next = j;
        }
      }
      l.rank[i] = (uint16_t)rank;
      l.next[i] = (uint16_t)next;
      l.count[i] = (uint16_t)(rank == 0 ? count : 0);
      frequent |= count >= kFrequent;
    }
    frequent = __syncthreads_or(frequent);
    const float4* row = dx + base * d4 + c;
    for (int i = w; i < m; i += kWarps) {
      if (l.count[i] == 0 || l.count[i] >= kFrequent) continue;
      float4 sum = zero;
      for (int e = i; e < m;) {
        float4 g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          g[u] = e < m && mine ? row[(int64_t)l.at[e] * d4] : zero;
          if (e < m) e = l.next[e];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) sum = sum + g[u];
      }
      if (mine) {
        float4* out = dtable + ((int64_t)l.key[i] * buckets + bucket) * d4 + c;
        *out = *out + sum;
      }
    }
    for (int i = 0; frequent && i < m; ++i) {
      const int count = l.count[i];
      if (count < kFrequent) continue;
      for (int j = threadIdx.x; j < m; j += kEmbThreads)
        if (l.key[j] == l.key[i]) l.rows[l.rank[j]] = l.at[j];
      __syncthreads();
      float4 sum = zero;
      for (int e = w; e < count; e += 8 * kWarps) {
        float4 g[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int at = e + u * kWarps;
          g[u] = at < count && mine ? row[(int64_t)l.rows[at] * d4] : zero;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) sum = sum + g[u];
      }
      l.part[w][lane] = sum;
      __syncthreads();
      if (w == 0 && mine) {
        sum = l.part[0][lane];
#pragma unroll
        for (int v = 1; v < kWarps; ++v) sum = sum + l.part[v][lane];
        float4* out = dtable + ((int64_t)l.key[i] * buckets + bucket) * d4 + c;
        *out = *out + sum;
      }
      // the next one writes `part` only behind its own first barrier
    }
    __syncthreads();  // the lists are used up; and a table row may go to another warp in the next round
  }
}

// The first `buckets` x `chunks` blocks do the tokens, the others the positions.
__global__ void __launch_bounds__(kEmbThreads)
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
  const int64_t chunks = (d4 + 31) / 32, position_blocks = (int64_t)seq * ((d4 + kEmbThreads - 1) / kEmbThreads);
  // As many token blocks as are resident, each of which looks through all tokens, but at least 8 tokens for one.
  int64_t buckets = (int64_t)sm_count * 5 / chunks;
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
