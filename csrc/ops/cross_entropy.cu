// Fused softmax cross-entropy over bf16 logits for the language-model head.
//   forward : one CTA per row, one pass (online max / sum-of-exponentials in fp32) -> per-row loss and
//             log-sum-exp; the 8192 x 50304 logits are read once and never widened to an fp32 tensor.
//   backward: dlogits = (exp(logit - lse) - [j == target]) * grad / rows, written in bf16 over the logits
//             (they are not needed afterwards); padding columns beyond the vocabulary get zero.
// Replaces the cast + log_softmax + nll_loss kernels (and their fp32 temporaries of rows x vocab) of an
// unfused loss.  No counterpart in the reference (it has no model code).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "mccl.h"
#include "mccl_ops.h"

namespace {

using namespace mccl;

// Small CTAs: several of them share an SM, so that the ends of rows (a last turn of the walk that few threads take, the fold of
// the CTA's sums) lie beside other rows' loads.  Backward with 512 threads / 256: 8192 x 50257 285 / 258 us (6.4 TB/s).
constexpr int kCeThreads = 256;
constexpr int kCeUnroll = 4;                   // 16-byte pieces in flight per thread in long rows: with one, the row's loads wait for each other
constexpr int64_t kIgnored = -100;             // the target value torch's cross-entropy leaves out

struct MaxSum { float m, s; };                 // running maximum and sum of exp(x - m)
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLowest = -3.402823466e38f;    // a maximum of nothing: below every finite bf16 number, and minus itself zero
__device__ __forceinline__ MaxSum combine(MaxSum a, MaxSum b) {
  const float m = fmaxf(a.m, b.m);
  return MaxSum{m, a.s * __expf(a.m - m) + b.s * __expf(b.m - m)};
}
__device__ __forceinline__ void unpack(const uint4& q, float* f) {
  const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int k = 0; k < 4; ++k) { const float2 t = __bfloat1622float2(e[k]); f[2 * k] = t.x; f[2 * k + 1] = t.y; }
}
// Values enter one after another: s = s exp(m - x) + 1 where x is a new maximum and s + exp(x - m) where not.  The maximum
// is subtracted before anything is scaled: exp(x - m) as 2^(x log2e - m log2e) would save an instruction, but it rounds
// m log2e (an error of |m| 2^-24 in every exponent) and overflows for logits near the type's lowest value, which masks are made
// of.
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ void add(MaxSum& a, bool up, float e) { a.s = up ? __fmaf_rn(a.s, e, 1.f) : __fadd_rn(a.s, e); }
__device__ __forceinline__ void push(MaxSum& a, float x) {
  add(a, x > a.m, ex2(-fabsf((x - a.m) * kLog2e)));
  a.m = fmaxf(a.m, x);
}
// Eight of them.  Instructions bound the forward pass here, at eight values of nine slots each a turn (8192 x 50257: 201 us):
// the eight maxima first, then differences and products two at a time, then the sums, predicated: 148 us, 5.6 TB/s.  (With a
// branch for a new maximum, which some lane of a warp takes nearly always: 254 us.)
__device__ __forceinline__ void push8(MaxSum& a, const uint4& q) {
  float f[8], m[9], e[8];
  unpack(q, f);
  m[0] = a.m;
#pragma unroll
  for (int k = 0; k < 8; ++k) m[k + 1] = fmaxf(m[k], f[k]);
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    float d0, d1;
    split((f2(f[k], f[k + 1]) + f2(-m[k], -m[k + 1])) * f2(kLog2e), &d0, &d1);
    e[k] = ex2(-fabsf(d0));
    e[k + 1] = ex2(-fabsf(d1));
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) add(a, f[k] > m[k], e[k]);
  a.m = m[8];
}

// The part of a row between its first and last 16-byte boundary: [head, head + 8 * vecs) of n elements.
struct Span { int head, vecs; };
__device__ __forceinline__ Span spanOf(const __nv_bfloat16* x, int n) {
  int head = (int)((16u - (uint32_t)(reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / 2;
  if (head > n) head = n;
  return Span{head, (n - head) / 8};
}

template <int U>
__global__ void __launch_bounds__(kCeThreads, 6) ceForwardKernel(const __nv_bfloat16* logits, int64_t ld, int vocab,
                                                              const int64_t* targets, float* loss, float* lse) {
  __shared__ MaxSum warpAcc[kCeThreads / 32];
  const int64_t row = blockIdx.x;
  const __nv_bfloat16* x = logits + row * ld;
  MaxSum acc{kLowest, 0.f};
  const Span sp = spanOf(x, vocab);
  const uint4* v = reinterpret_cast<const uint4*>(x + sp.head);
  for (int i = threadIdx.x; i < sp.vecs; i += U * kCeThreads) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (i + u * kCeThreads < sp.vecs) q[u] = v[i + u * kCeThreads];
#pragma unroll
    for (int u = 0; u < U; ++u) if (i + u * kCeThreads < sp.vecs) push8(acc, q[u]);
  }
  const int tail = sp.head + sp.vecs * 8;
  if ((int)threadIdx.x < sp.head) push(acc, __bfloat162float(x[threadIdx.x]));
  if (tail + (int)threadIdx.x < vocab) push(acc, __bfloat162float(x[tail + threadIdx.x]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum other{__shfl_xor_sync(0xffffffffu, acc.m, o), __shfl_xor_sync(0xffffffffu, acc.s, o)};
    acc = combine(acc, other);
  }
  if ((threadIdx.x & 31) == 0) warpAcc[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    MaxSum t = warpAcc[0];
    for (int w = 1; w < kCeThreads / 32; ++w) t = combine(t, warpAcc[w]);
    const float l = t.m == INFINITY ? __int_as_float(0x7fffffff) : t.m + logf(t.s);      // inf - inf in the exponent
    const int64_t tgt = targets[row];
    lse[row] = l;
    loss[row] = (tgt >= 0 && tgt < vocab) ? l - __bfloat162float(x[tgt]) : 0.f;     // out-of-range target: ignored row
  }
}

// Mean over the rows' losses, in a fixed order: over all rows or, with `targets`, over those whose target is a column
// (`inverse`: one over their number, for the backward pass); there a target that is neither a column nor kIgnored makes the
// mean NaN.
__global__ void __launch_bounds__(1024) meanKernel(const float* v, int64_t n, const int64_t* targets, int vocab, float* out, float* inverse) {
  __shared__ float acc[32];
  __shared__ int used;
  if (threadIdx.x == 0) used = 0;
  __syncthreads();
  float t = 0.f;
  int c = 0;
  for (int64_t i = threadIdx.x; i < n; i += 8 * 1024) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = i + u * 1024 < n ? v[i + u * 1024] : 0.f;
    if (targets != nullptr)
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (i + u * 1024 >= n) continue;
        const int64_t k = targets[i + u * 1024];
        if (k >= 0 && k < vocab) ++c;
        else if (k != kIgnored) x[u] = __int_as_float(0x7fffffff);
      }
    t += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  }
  if (targets != nullptr) atomicAdd(&used, c);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) acc[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  t = acc[threadIdx.x];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x != 0) return;
  const float rows = targets != nullptr ? (float)used : (float)n;
  *out = t / rows;
  if (inverse != nullptr) *inverse = 1.f / rows;
}

// Reads and writes every logit once: 8192 x 50257 307 us with one piece in flight, 259 us with four.
// blockIdx.y: which slice of the row (one unless there are few rows).  The last rows come first: they are what the forward
// pass, or the projection, left in L2.
template <int U>
__global__ void __launch_bounds__(kCeThreads) ceBackwardKernel(__nv_bfloat16* logits, int64_t ld, int vocab, int width,
                                                               const int64_t* targets, const float* lse, const float* gradOut,
                                                               const float* inverse, float invRows) {
  const int64_t row = (int64_t)gridDim.x - 1 - blockIdx.x;
  __nv_bfloat16* x = logits + row * ld;
  const float l = lse[row];
  const int64_t tgt64 = targets[row];
  const bool live = tgt64 >= 0 && tgt64 < vocab;
  const int tgt = live ? (int)tgt64 : -1;
  const float scale = live ? (*gradOut) * (inverse != nullptr ? *inverse : invRows) : 0.f;
  auto one = [&](int j, float xj) -> float {
    if (j >= vocab) return 0.f;
    return (__expf(xj - l) - (j == tgt ? 1.f : 0.f)) * scale;
  };
  const Span sp = spanOf(x, width);
  uint4* v = reinterpret_cast<uint4*>(x + sp.head);
  const int stride = (int)gridDim.y * kCeThreads;
  for (int i = (int)blockIdx.y * kCeThreads + threadIdx.x; i < sp.vecs; i += U * stride) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (i + u * stride < sp.vecs) q[u] = v[i + u * stride];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i + u * stride >= sp.vecs) continue;
      const int j0 = sp.head + (i + u * stride) * 8;
      float f[8];
      unpack(q[u], f);
      if (j0 + 8 <= vocab && (unsigned)(tgt - j0) >= 8u) {       // neither the target nor padding in these eight
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = __expf(f[k] - l) * scale;
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = one(j0 + k, f[k]);
      }
      __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&q[u]);
#pragma unroll
      for (int k = 0; k < 4; ++k) e[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
      v[i + u * stride] = q[u];
    }
  }
  if (blockIdx.y == 0) {
    const int tail = sp.head + sp.vecs * 8, h = threadIdx.x, t = tail + (int)threadIdx.x;
    if (h < sp.head) x[h] = __float2bfloat16_rn(one(h, __bfloat162float(x[h])));
    if (t < width) x[t] = __float2bfloat16_rn(one(t, __bfloat162float(x[t])));
  }
}

// Rows that 256 threads walk in two turns or fewer take the form with one piece in flight: fewer registers, so more
// rows a SM (16384 x 1000 forward 47 -> 39 us, backward 41 -> 30 us).
bool shortRow(int n) { return n <= 2 * 8 * kCeThreads; }

// CTAs per row in the backward pass: few rows are shared by up to eight CTAs each, as long as there are no more than six CTAs an SM and each keeps
// 4096 elements (two turns of its loads).
int ceSplit(int64_t rows, int n) {
  int r = 1;
  while (r < 8 && rows * r * 2 <= 148 * 6 && n / (r * 2) >= 4096) r *= 2;
  return r;
}

}  // namespace

// loss[row] = logsumexp(logits[row, :vocab]) - logits[row, target[row]]; lse[row] keeps the log-sum-exp.
extern "C" mcclResult_t mcclCrossEntropyForward(const void* logits, int64_t rows, int64_t ld, int vocab, const int64_t* targets,
                                                float* loss, float* lse, mcclStream_t stream) {
  if (logits == nullptr || targets == nullptr || loss == nullptr || lse == nullptr || rows < 0 || vocab <= 0 || ld < vocab)
    return mcclInvalidArgument;
  if (rows == 0) return mcclSuccess;
  auto* kernel = shortRow(vocab) ? ceForwardKernel<1> : ceForwardKernel<kCeUnroll>;
  kernel<<<(unsigned)rows, kCeThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(logits), ld, vocab,
                                                                                   targets, loss, lse);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

// The same followed by the mean of the rows' losses in *mean: over all rows, or with `inverse` over the rows whose target is
// a column, one over whose number goes there.
extern "C" mcclResult_t mcclCrossEntropyMean(const void* logits, int64_t rows, int64_t ld, int vocab, const int64_t* targets, float* loss,
                                             float* lse, float* mean, float* inverse, mcclStream_t stream) {
  if (mean == nullptr) return mcclInvalidArgument;
  const mcclResult_t rc = mcclCrossEntropyForward(logits, rows, ld, vocab, targets, loss, lse, stream);
  if (rc != mcclSuccess) return rc;
  meanKernel<<<1, 1024, 0, reinterpret_cast<cudaStream_t>(stream)>>>(loss, rows, inverse != nullptr ? targets : nullptr, vocab, mean, inverse);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

// In place: logits[row, j] <- d(mean loss)/d(logit) * gradOut for j < vocab, 0 for vocab <= j < width.  inverse: what
// mcclCrossEntropyMean stored there, or null where the mean was over all rows.
extern "C" mcclResult_t mcclCrossEntropyMeanBackward(void* logits, int64_t rows, int64_t ld, int vocab, int width, const int64_t* targets,
                                                     const float* lse, const float* gradOut, const float* inverse, mcclStream_t stream) {
  if (logits == nullptr || targets == nullptr || lse == nullptr || gradOut == nullptr || rows < 0 || vocab <= 0 || width < vocab ||
      ld < width) return mcclInvalidArgument;
  if (rows == 0) return mcclSuccess;
  auto* kernel = shortRow(width) ? ceBackwardKernel<1> : ceBackwardKernel<kCeUnroll>;
  kernel<<<dim3((unsigned)rows, (unsigned)ceSplit(rows, width)), kCeThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(logits), ld, vocab, width, targets, lse, gradOut, inverse, 1.0f / (float)rows);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

extern "C" mcclResult_t mcclCrossEntropyBackward(void* logits, int64_t rows, int64_t ld, int vocab, int width, const int64_t* targets,
                                                 const float* lse, const float* gradOut, mcclStream_t stream) {
  return mcclCrossEntropyMeanBackward(logits, rows, ld, vocab, width, targets, lse, gradOut, nullptr, stream);
}
