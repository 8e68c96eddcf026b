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
constexpr int kMaxTokens = 16384;             // of the backward pass: a token that occurs again scans all of them
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

// One CTA per token.  A token that occurs once adds its row.  Of one that occurs again, the first occurrence adds the sum of
// all rows in token order (a fixed order, in fp32), which it finds by scanning the indices; the others leave as soon as the
// scan shows them an earlier one.
template <int VPT>
__global__ void __launch_bounds__(kEmbThreads) tableGradKernel(const int64_t* idx, const uint4* dy, const int* count, int n, int64_t vocab,
                                                               int vecs, uint4* grad) {
  __shared__ int found[kEmbThreads];
  __shared__ int warpFound[kEmbThreads / 32];
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
    int seen = 0;
    for (int base = 0; base < n && seen < all; base += kEmbThreads) {
      const bool hit = base + tid < n && idx[base + tid] == id;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) warpFound[warp] = __popc(m);
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int w = 0; w < kEmbThreads / 32; ++w) { if (w < warp) before += warpFound[w]; total += warpFound[w]; }
      if (hit) found[before + __popc(m & ((1u << lane) - 1u))] = base + tid;
      __syncthreads();
      if (total > 0 && seen == 0 && found[0] != t) return;       // an earlier occurrence does the work
      for (int k = seen == 0 ? 1 : 0; k < total; k += 4) {
        uint4 q[4][VPT];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < VPT; ++j) {
            const int v = tid + j * kEmbThreads;
            q[u][j] = k + u < total && v < vecs ? dy[(int64_t)found[k + u] * vecs + v] : make_uint4(0, 0, 0, 0);
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < VPT; ++j) {
            float f[8];
            unpack(q[u][j], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[j][e] += f[e];
          }
      }
      seen += total;
      __syncthreads();
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

// tableGrad rows += the rows of dy with their index; posGrad (may be null) += dy summed over the batch.  count: vocab ints of work memory.
mcclResult_t mcclEmbeddingBackward(const int64_t* idx, const void* dy, void* tableGrad, void* posGrad, int32_t* count, int64_t tokens, int seq,
                                   int64_t vocab, int D, mcclStream_t stream) {
  if (!idx || !dy || !tableGrad || !count || tokens <= 0 || tokens > kMaxTokens || seq <= 0 || tokens % seq || D <= 0 || D % 8 ||
      D / 8 > kMaxVecs || !aligned16(dy) || !aligned16(tableGrad) || !aligned16(posGrad)) return mcclInvalidArgument;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int n = (int)tokens, vecs = D / 8;
  const uint4* g = static_cast<const uint4*>(dy);
  uint4* tg = static_cast<uint4*>(tableGrad);
  if (cudaMemsetAsync(count, 0, vocab * sizeof(int32_t), s) != cudaSuccess) return mcclSystemError;
  countTokensKernel<<<(n + 255) / 256, 256, 0, s>>>(idx, n, vocab, count);
  if (vecs <= kEmbThreads) tableGradKernel<1><<<n, kEmbThreads, 0, s>>>(idx, g, count, n, vocab, vecs, tg);
  else if (vecs <= 2 * kEmbThreads) tableGradKernel<2><<<n, kEmbThreads, 0, s>>>(idx, g, count, n, vocab, vecs, tg);
  else tableGradKernel<4><<<n, kEmbThreads, 0, s>>>(idx, g, count, n, vocab, vecs, tg);
  const int64_t perSeq = (int64_t)seq * vecs;
  if (posGrad != nullptr) posGradKernel<<<(unsigned)((perSeq + 255) / 256), 256, 0, s>>>(g, n / seq, perSeq, static_cast<uint4*>(posGrad));
  return launchedOk();
}

}  // extern "C"
