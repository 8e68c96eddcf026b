// Token and position embedding of a decoder: one pass forward, and a backward pass that adds into the gradient of the table
// only the rows that occur (a dense gradient of a 50304 x 1024 table is 103 MB to clear, to scatter into and to add).
// No counterpart in the reference (it has no model code).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mccl.h"
#include "mccl_ops.h"

namespace {

constexpr int kEmbThreads = 128;
constexpr int kMaxTokens = 16384;             // of the backward pass: every token that occurs in two chunks is looked for in all of them
constexpr int kMaxVecs = 4 * kEmbThreads;     // 16-byte pieces of a row: D <= 4096

__device__ __forceinline__ void unpack(const uint4& q, float* f) {
  const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int k = 0; k < 4; ++k) { const float2 t = __bfloat1622float2(e[k]); f[2 * k] = t.x; f[2 * k + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack(const float* f) {
  uint4 q;
  __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int k = 0; k < 4; ++k) e[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
  return q;
}

// out[t] = table[idx[t]] + pos[t % seq] (pos may be null); NaN for an index outside the table.
__global__ void __launch_bounds__(256) embedKernel(const int64_t* idx, const uint4* table, const uint4* pos, int64_t n, int seq,
                                                   int64_t vocab, int vecs, uint4* out) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n * vecs) return;
  const int64_t t = i / vecs;
  const int v = (int)(i - t * vecs);
  const int64_t id = idx[t];
  float a[8], b[8];
  unpack(pos != nullptr ? pos[(t % seq) * vecs + v] : make_uint4(0, 0, 0, 0), b);
  if (id >= 0 && id < vocab) {
    unpack(table[id * vecs + v], a);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] += b[k];
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = __int_as_float(0x7fffffff);
  }
  out[i] = pack(a);
}

__global__ void countTokensKernel(const int64_t* idx, int n, int64_t vocab, int* count) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n && idx[t] >= 0 && idx[t] < vocab) atomicAdd(&count[idx[t]], 1);
}

constexpr int kChunk = kEmbThreads;           // tokens that one CTA adds up
constexpr int kMaxChunks = kMaxTokens / kChunk;
constexpr int kScan = 8;                      // chunks looked through at once

// acc += row r of a [*, vecs] matrix for every r of `list` in its order, four rows in flight; fp32 rows (two pieces) or bf16.
template <int VPT, bool F32>
__device__ __forceinline__ void addRows(float (*acc)[8], const uint4* rows, const int* list, int from, int n, int vecs) {
  constexpr int P = F32 ? 2 : 1;
  for (int k = from; k < n; k += 4) {
    uint4 q[4][VPT][P];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        const int v = threadIdx.x + j * kEmbThreads;
#pragma unroll
        for (int p = 0; p < P; ++p)
          q[u][j][p] = k + u < n && v < vecs ? __ldcg(rows + ((int64_t)list[k + u] * vecs + v) * P + p) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        float f[8];
        if (F32) {
#pragma unroll
          for (int p = 0; p < P; ++p) {
            f[4 * p] = __uint_as_float(q[u][j][p].x); f[4 * p + 1] = __uint_as_float(q[u][j][p].y);
            f[4 * p + 2] = __uint_as_float(q[u][j][p].z); f[4 * p + 3] = __uint_as_float(q[u][j][p].w);
          }
        } else {
          unpack(q[u][j][0], f);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[j][e] += f[e];
      }
  }
}

// One CTA per token.  A token that occurs once adds its row.  Of one that occurs again, the first of a chunk of 128 tokens adds up the
// rows in the chunk; if there are others elsewhere the sum stays in fp32 at its place in `partial`, and the CTA that finds all
// of the token's rows done adds the chunks' sums, in token order whoever it is, so the result does not depend on the order of
// arrival.  Bound by the rows' memory (2 bytes an element) and, for a token that fills the batch, by 32 turns of a chunk and
// 32 of the chunks' sums; with one CTA for all rows of a token 16384 equal ones were 4096 turns.
template <int VPT>
__global__ void __launch_bounds__(kEmbThreads) tableGradKernel(const int64_t* idx, const uint4* dy, const int* count, int* done, uint4* partial,
                                                               int n, int64_t vocab, int vecs, uint4* grad) {
  constexpr int W = kEmbThreads / 32;
  __shared__ int found[kMaxChunks > kChunk ? kMaxChunks : kChunk];
  __shared__ unsigned hits[kScan][W];
  __shared__ int arrived;
  const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t id = idx[t];
  if (id < 0 || id >= vocab) return;
  float acc[VPT][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int v = tid + j * kEmbThreads;
    unpack(v < vecs ? dy[(int64_t)t * vecs + v] : make_uint4(0, 0, 0, 0), acc[j]);
  }
  const int all = count[id];
  if (all > 1) {
    const int base = t / kChunk * kChunk;
    const bool hit = base + tid < n && idx[base + tid] == id;
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) hits[0][warp] = m;
    __syncthreads();
    int before = 0, here = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) { const int c = __popc(hits[0][w]); if (w < warp) before += c; here += c; }
    if (hit) found[before + __popc(m & ((1u << lane) - 1u))] = base + tid;
    __syncthreads();
    if (found[0] != t) return;                                       // an earlier one of the chunk does the work
    addRows<VPT, false>(acc, dy, found, 1, here, vecs);
    if (here < all) {
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        const int v = tid + j * kEmbThreads;
        if (v >= vecs) continue;
        float4* to = reinterpret_cast<float4*>(partial + ((int64_t)t * vecs + v) * 2);
        to[0] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        to[1] = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
      }
      __threadfence();
      __syncthreads();
      if (tid == 0) arrived = atomicAdd(&done[id], here) + here;
      __syncthreads();
      if (arrived < all) return;                                     // whoever completes the count adds up
      __threadfence();
      int firsts = 0;                                                // the first token of this kind in every chunk
      for (int c0 = 0; c0 * kChunk < n; c0 += kScan) {
#pragma unroll
        for (int u = 0; u < kScan; ++u) {
          const int i = (c0 + u) * kChunk + tid;
          const unsigned b = __ballot_sync(0xffffffffu, i < n && idx[i] == id);
          if (lane == 0) hits[u][warp] = b;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kScan; ++u) {
          int first = -1;
#pragma unroll
          for (int w = W - 1; w >= 0; --w) if (hits[u][w]) first = w * 32 + __ffs(hits[u][w]) - 1;
          if (first >= 0) { if (tid == 0) found[firsts] = (c0 + u) * kChunk + first; ++firsts; }
        }
        __syncthreads();
      }
#pragma unroll
      for (int j = 0; j < VPT; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[j][e] = 0.f;
      addRows<VPT, true>(acc, partial, found, 0, firsts, vecs);
    }
  }
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int v = tid + j * kEmbThreads;
    if (v >= vecs) continue;
    float f[8];
    unpack(grad[id * vecs + v], f);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] += __bfloat162float(__float2bfloat16_rn(acc[j][e]));      // rounded as a gradient of its own is
    grad[id * vecs + v] = pack(f);
  }
}

// grad[s] += sum over the batch of dy[b][s].
__global__ void __launch_bounds__(256) posGradKernel(const uint4* dy, int batch, int64_t perSeq, uint4* grad) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= perSeq) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int b0 = 0; b0 < batch; b0 += 4) {
    uint4 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) q[u] = b0 + u < batch ? dy[(b0 + u) * perSeq + i] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float f[8];
      unpack(q[u], f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += f[e];
    }
  }
  float f[8];
  unpack(grad[i], f);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] += acc[e];
  grad[i] = pack(f);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
mcclResult_t launchedOk() { return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError; }

}  // namespace

extern "C" {

mcclResult_t mcclEmbeddingForward(const int64_t* idx, const void* table, const void* pos, void* out, int64_t tokens, int seq, int64_t vocab,
                                  int D, mcclStream_t stream) {
  if (!idx || !table || !out || tokens <= 0 || seq <= 0 || D <= 0 || D % 8 || !aligned16(table) || !aligned16(pos) || !aligned16(out))
    return mcclInvalidArgument;
  embedKernel<<<(unsigned)((tokens * (D / 8) + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      idx, static_cast<const uint4*>(table), static_cast<const uint4*>(pos), tokens, seq, vocab, D / 8, static_cast<uint4*>(out));
  return launchedOk();
}

int mcclEmbeddingMaxTokens(void) { return kMaxTokens; }

// Bytes of work memory of the function below.
int64_t mcclEmbeddingWork(int64_t tokens, int64_t vocab, int D) {
  return (2 * vocab * (int64_t)sizeof(int32_t) + 15) / 16 * 16 + tokens * D * (int64_t)sizeof(float);
}

// tableGrad rows += the rows of dy with their index; posGrad (may be null) += dy summed over the batch.  work: 16-byte aligned.
mcclResult_t mcclEmbeddingBackwardWork(const int64_t* idx, const void* dy, void* tableGrad, void* posGrad, void* work, int64_t tokens, int seq,
                                       int64_t vocab, int D, mcclStream_t stream) {
  if (!idx || !dy || !tableGrad || !work || tokens <= 0 || tokens > kMaxTokens || seq <= 0 || tokens % seq || D <= 0 || D % 8 || vocab <= 0 ||
      D / 8 > kMaxVecs || !aligned16(dy) || !aligned16(tableGrad) || !aligned16(posGrad) || !aligned16(work)) return mcclInvalidArgument;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int n = (int)tokens, vecs = D / 8;
  const uint4* g = static_cast<const uint4*>(dy);
  uint4* tg = static_cast<uint4*>(tableGrad);
  int* count = static_cast<int*>(work);
  int* done = count + vocab;
  uint4* partial = reinterpret_cast<uint4*>(static_cast<char*>(work) + (2 * vocab * (int64_t)sizeof(int32_t) + 15) / 16 * 16);
  if (cudaMemsetAsync(count, 0, 2 * vocab * sizeof(int32_t), s) != cudaSuccess) return mcclSystemError;
  countTokensKernel<<<(n + 255) / 256, 256, 0, s>>>(idx, n, vocab, count);
  if (vecs <= kEmbThreads) tableGradKernel<1><<<n, kEmbThreads, 0, s>>>(idx, g, count, done, partial, n, vocab, vecs, tg);
  else if (vecs <= 2 * kEmbThreads) tableGradKernel<2><<<n, kEmbThreads, 0, s>>>(idx, g, count, done, partial, n, vocab, vecs, tg);
  else tableGradKernel<4><<<n, kEmbThreads, 0, s>>>(idx, g, count, done, partial, n, vocab, vecs, tg);
  const int64_t perSeq = (int64_t)seq * vecs;
  if (posGrad != nullptr) posGradKernel<<<(unsigned)((perSeq + 255) / 256), 256, 0, s>>>(g, n / seq, perSeq, static_cast<uint4*>(posGrad));
  return launchedOk();
}

// The same with work memory of its own, allocated and freed in the stream's order; count: not used.
mcclResult_t mcclEmbeddingBackward(const int64_t* idx, const void* dy, void* tableGrad, void* posGrad, int32_t* count, int64_t tokens, int seq,
                                   int64_t vocab, int D, mcclStream_t stream) {
  if (!count || tokens <= 0 || tokens > kMaxTokens || vocab <= 0 || D <= 0 || D / 8 > kMaxVecs) return mcclInvalidArgument;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  void* work = nullptr;
  if (cudaMallocAsync(&work, mcclEmbeddingWork(tokens, vocab, D), s) != cudaSuccess) { cudaGetLastError(); return mcclSystemError; }
  const mcclResult_t rc = mcclEmbeddingBackwardWork(idx, dy, tableGrad, posGrad, work, tokens, seq, vocab, D, stream);
  return cudaFreeAsync(work, s) == cudaSuccess ? rc : mcclSystemError;
}

}  // extern "C"
