// Expert routing and the token movement of a mixture-of-experts layer whose experts are all on this GPU.
//   route    softmax over the experts in fp32, top-1 expert (the lowest index of equals), its probability as the gate, and
//            the token's slot among the tokens of its expert in token order.  Two small launches: chunks of 256 tokens count
//            their experts, then every chunk adds the counts of the chunks before it.  (A cumulative sum over a [tokens,
//            experts] one-hot matrix of 64-bit integers, as a tensor library does it, took 1.7 ms for 8192 tokens.)
//   gather / scatter  written from the side of the slots, so that a slot is written once, by a copy or by zeros, and
//            nothing has to be cleared before.
// Bound by memory, a row of the activations read or written per token and direction.
// No counterpart in the reference (its AllToAll has no routing).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mccl.h"
#include "mccl_ops.h"

namespace {

constexpr int kChunk = 256;                    // tokens per CTA of the routing kernels
constexpr int kMaxExperts = 1024;
constexpr int kRowThreads = 256, kRowWarps = kRowThreads / 32;

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
__device__ __forceinline__ float rounded(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// gate[t] = bf16(p of the best expert), lse[t]; flat[t] = expert << 8 | rank among this chunk's tokens of the expert;
// hist[chunk][expert] = tokens of the chunk.
__global__ void __launch_bounds__(kChunk) routeCountKernel(const __nv_bfloat16* logits, int T, int E, float* gate, float* lse, int* flat, int* hist) {
  extern __shared__ int counts[];              // [warps][E]
  constexpr int W = kChunk / 32;
  for (int i = threadIdx.x; i < W * E; i += kChunk) counts[i] = 0;
  __syncthreads();
  const int t = blockIdx.x * kChunk + threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int best = -1;
  if (t < T) {
    const __nv_bfloat16* x = logits + (int64_t)t * E;
    float m = -INFINITY;
    best = 0;
    for (int e = 0; e < E; ++e) { const float v = __bfloat162float(x[e]); if (v > m) { m = v; best = e; } }
    float s = 0.f;
    for (int e = 0; e < E; ++e) s += expf(__bfloat162float(x[e]) - m);
    gate[t] = rounded(1.f / s);
    lse[t] = m + logf(s);
  }
  // Rank inside the warp, then the warps in order.
  const unsigned same = __match_any_sync(0xffffffffu, best);
  const int inWarp = __popc(same & ((1u << lane) - 1u));
  if (best >= 0 && inWarp == 0) counts[warp * E + best] = __popc(same);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kChunk) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) { const int c = counts[w * E + e]; counts[w * E + e] = run; run += c; }
    hist[(int64_t)blockIdx.x * E + e] = run;
  }
  __syncthreads();
  if (t < T) flat[t] = best << 8 | (counts[warp * E + best] + inWarp);
}

// flat[t] -> expert * capacity + slot, or -1 beyond the capacity; inverse[slot] = t and kept[expert] = slots filled, both
// when wanted.
__global__ void __launch_bounds__(kChunk) routeSlotKernel(int T, int E, int capacity, const int* hist, int* flat, int* inverse, int* kept) {
  extern __shared__ int base[];                // [E]
  const int chunk = blockIdx.x;
  // Several threads share an expert's sum over the chunks before this one.
  for (int e = threadIdx.x; e < E; e += kChunk) base[e] = 0;
  __syncthreads();
  const int per = E < kChunk ? kChunk / E : 1, e0 = threadIdx.x % E, part = threadIdx.x / E;
  if (E >= kChunk || part < per) {
    for (int e = E >= kChunk ? threadIdx.x : e0; e < E; e += kChunk) {
      int s = 0;
      for (int c = E >= kChunk ? 0 : part; c < chunk; c += per) s += hist[(int64_t)c * E + e];
      if (s) atomicAdd(&base[e], s);           // whole numbers: the order does not matter
    }
  }
  __syncthreads();
  const int t = chunk * kChunk + threadIdx.x;
  if (t < T) {
    const int v = flat[t], e = v >> 8, slot = base[e] + (v & 255);
    const int f = slot < capacity ? e * capacity + slot : -1;
    flat[t] = f;
    if (inverse != nullptr && f >= 0) inverse[f] = t;
  }
  if (kept != nullptr && chunk == (int)gridDim.x - 1)
    for (int e = threadIdx.x; e < E; e += kChunk) {
      const int all = base[e] + hist[(int64_t)chunk * E + e];
      kept[e] = all < capacity ? all : capacity;
    }
}

// One warp per slot: slots[s] = rows[inverse[s]], or zero where the slot is empty.
__global__ void __launch_bounds__(kRowThreads) fillSlotsKernel(const uint4* rows, const int* inverse, const int* kept, int E, int capacity,
                                                               int vecs, uint4* slots) {
  const int64_t s = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (s >= (int64_t)E * capacity) return;
  const int e = (int)(s / capacity), lane = threadIdx.x & 31;
  const bool full = (int)(s - (int64_t)e * capacity) < kept[e];
  const uint4* src = rows + (full ? (int64_t)inverse[s] * vecs : 0);
  uint4* dst = slots + s * vecs;
  constexpr int U = 4;
  for (int v0 = lane; v0 < vecs; v0 += 32 * U) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = full && v0 + 32 * u < vecs ? src[v0 + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) if (v0 + 32 * u < vecs) dst[v0 + 32 * u] = q[u];
  }
}

// One warp per token: out[t] = gate[t] * slots[flat[t]], zero for a dropped token.
__global__ void __launch_bounds__(kRowThreads) combineKernel(const uint4* slots, const int* flat, const float* gate, int T, int vecs, uint4* out) {
  const int t = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (t >= T) return;
  const int f = flat[t], lane = threadIdx.x & 31;
  const uint4* src = slots + (int64_t)(f < 0 ? 0 : f) * vecs;
  const float g = gate[t];
  uint4* dst = out + (int64_t)t * vecs;
  constexpr int U = 4;
  for (int v0 = lane; v0 < vecs; v0 += 32 * U) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = f >= 0 && v0 + 32 * u < vecs ? src[v0 + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (v0 + 32 * u >= vecs) continue;
      float x[8];
      unpack(q[u], x);
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] *= g;
      dst[v0 + 32 * u] = pack(x);
    }
  }
}

// One warp per slot: dslots[s] = gate[t] * dy[t] and dgate[t] = <dy[t], slots[s]> for the token t in the slot; zero rows
// where it is empty.
__global__ void __launch_bounds__(kRowThreads) combineBackwardKernel(const uint4* dy, const uint4* slots, const int* inverse, const int* kept,
                                                                     const float* gate, int E, int capacity, int vecs, uint4* dslots,
                                                                     float* dgate) {
  const int64_t s = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (s >= (int64_t)E * capacity) return;
  const int e = (int)(s / capacity), lane = threadIdx.x & 31;
  const bool full = (int)(s - (int64_t)e * capacity) < kept[e];
  const int t = full ? inverse[s] : 0;
  const float g = full ? gate[t] : 0.f;
  const uint4 *dyr = dy + (int64_t)t * vecs, *row = slots + s * vecs;
  uint4* dst = dslots + s * vecs;
  float dot = 0.f;
  constexpr int U = 4;
  for (int v0 = lane; v0 < vecs; v0 += 32 * U) {
    uint4 q[U], p[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = full && v0 + 32 * u < vecs;
      q[u] = in ? dyr[v0 + 32 * u] : make_uint4(0, 0, 0, 0);
      p[u] = in ? row[v0 + 32 * u] : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (v0 + 32 * u >= vecs) continue;
      float x[8], y[8];
      unpack(q[u], x);
      unpack(p[u], y);
#pragma unroll
      for (int k = 0; k < 8; ++k) { dot += x[k] * y[k]; x[k] *= g; }
      dst[v0 + 32 * u] = pack(x);
    }
  }
  dot = warpSum(dot);
  if (full && lane == 0) dgate[t] = dot;
}

// Gradient of the tokens: the row that comes back from the expert and what flows through the router,
//   dlogits[t][e] = p[e] * ((e == expert) - p[expert]) * dgate[t]      (zero for a dropped token: its output is zero)
//   dx[t] = dslots[flat[t]] + sum over e of dlogits[t][e] * router[e].
// A warp takes four tokens at a time, so that a piece of the router's weight is read once for the four of them; more experts
// than the sum is worth doing here for (router null) leave it to a matrix product.
constexpr int kTok = 4;
__global__ void __launch_bounds__(kRowThreads) tokenBackwardKernel(const uint4* dslots, const int* flat, const float* dgate,
                                                                   const __nv_bfloat16* logits, const float* lse, const uint4* router,
                                                                   int T, int E, int capacity, int vecs, __nv_bfloat16* dlogits, uint4* dx) {
  extern __shared__ float sh[];                // [warps][E][kTok]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (blockIdx.x * kRowWarps + warp) * kTok;
  if (t0 >= T) return;
  float* dl = sh + warp * E * kTok;
  int f[kTok];
#pragma unroll
  for (int i = 0; i < kTok; ++i) f[i] = t0 + i < T ? flat[t0 + i] : -1;
#pragma unroll
  for (int i = 0; i < kTok; ++i) {
    if (t0 + i >= T) { for (int e = lane; e < E; e += 32) dl[e * kTok + i] = 0.f; continue; }
    const __nv_bfloat16* x = logits + (int64_t)(t0 + i) * E;
    const int best = f[i] < 0 ? 0 : f[i] / capacity;
    const float l = lse[t0 + i], dg = f[i] < 0 ? 0.f : rounded(dgate[t0 + i]);
    const float pb = expf(__bfloat162float(x[best]) - l);
    for (int e = lane; e < E; e += 32) {
      const float p = expf(__bfloat162float(x[e]) - l);
      const float d = rounded(p * ((e == best ? dg : 0.f) - pb * dg));
      dl[e * kTok + i] = d;
      dlogits[(int64_t)(t0 + i) * E + e] = __float2bfloat16_rn(d);
    }
  }
  __syncwarp();
  for (int v = lane; v < vecs; v += 32) {
    float acc[kTok][8];
#pragma unroll
    for (int i = 0; i < kTok; ++i) unpack(f[i] >= 0 ? dslots[(int64_t)f[i] * vecs + v] : make_uint4(0, 0, 0, 0), acc[i]);
    if (router != nullptr) {
#pragma unroll 4
      for (int e = 0; e < E; ++e) {
        float w[8];
        unpack(router[(int64_t)e * vecs + v], w);
        const float4 d = *reinterpret_cast<const float4*>(dl + e * kTok);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          acc[0][k] += d.x * w[k]; acc[1][k] += d.y * w[k]; acc[2][k] += d.z * w[k]; acc[3][k] += d.w * w[k];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kTok; ++i) if (t0 + i < T) dx[(int64_t)(t0 + i) * vecs + v] = pack(acc[i]);
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
mcclResult_t launchedOk() { return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError; }
unsigned rowBlocks(int64_t rows) { return (unsigned)((rows + kRowWarps - 1) / kRowWarps); }

}  // namespace

extern "C" {

int mcclMoeRouteMaxExperts(void) { return kMaxExperts; }

// Ints of work memory mcclMoeRoute needs.
int64_t mcclMoeRouteScratch(int tokens, int experts) { return (int64_t)((tokens + kChunk - 1) / kChunk) * experts; }

mcclResult_t mcclMoeRoute(const void* logits, int tokens, int experts, int capacity, float* gate, float* lse, int32_t* flat,
                          int32_t* inverse, int32_t* kept, int32_t* scratch, mcclStream_t stream) {
  if (tokens < 0 || experts <= 0 || experts > kMaxExperts || capacity <= 0 || (int64_t)experts * capacity > INT32_MAX) return mcclInvalidArgument;
  if (tokens > 0 && (!logits || !gate || !lse || !flat || !scratch)) return mcclInvalidArgument;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (tokens == 0) return kept == nullptr || cudaMemsetAsync(kept, 0, experts * sizeof(int32_t), s) == cudaSuccess ? mcclSuccess : mcclSystemError;
  const unsigned chunks = (unsigned)((tokens + kChunk - 1) / kChunk);
  routeCountKernel<<<chunks, kChunk, kChunk / 32 * experts * sizeof(int), s>>>(static_cast<const __nv_bfloat16*>(logits), tokens, experts,
                                                                              gate, lse, flat, scratch);
  routeSlotKernel<<<chunks, kChunk, experts * sizeof(int), s>>>(tokens, experts, capacity, scratch, flat, inverse, kept);
  return launchedOk();
}

mcclResult_t mcclMoeFillSlots(const void* rows, const int32_t* inverse, const int32_t* kept, void* slots, int experts, int capacity,
                              int d, mcclStream_t stream) {
  if (!inverse || !kept || !slots || d <= 0 || d % 8 || !aligned16(rows) || !aligned16(slots)) return mcclInvalidArgument;
  fillSlotsKernel<<<rowBlocks((int64_t)experts * capacity), kRowThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(rows), inverse, kept, experts, capacity, d / 8, static_cast<uint4*>(slots));
  return launchedOk();
}

mcclResult_t mcclMoeCombine(const void* slots, const int32_t* flat, const float* gate, void* out, int tokens, int d, mcclStream_t stream) {
  if (d <= 0 || d % 8 || !aligned16(slots) || !aligned16(out)) return mcclInvalidArgument;
  if (tokens == 0) return mcclSuccess;
  combineKernel<<<rowBlocks(tokens), kRowThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(static_cast<const uint4*>(slots), flat, gate,
                                                                                              tokens, d / 8, static_cast<uint4*>(out));
  return launchedOk();
}

mcclResult_t mcclMoeCombineBackward(const void* dy, const void* slots, const int32_t* inverse, const int32_t* kept, const float* gate,
                                    void* dslots, float* dgate, int experts, int capacity, int d, mcclStream_t stream) {
  if (!inverse || !kept || d <= 0 || d % 8 || !aligned16(dy) || !aligned16(slots) || !aligned16(dslots)) return mcclInvalidArgument;
  combineBackwardKernel<<<rowBlocks((int64_t)experts * capacity), kRowThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(dy), static_cast<const uint4*>(slots), inverse, kept, gate, experts, capacity, d / 8,
      static_cast<uint4*>(dslots), dgate);
  return launchedOk();
}

mcclResult_t mcclMoeTokenBackward(const void* dslots, const int32_t* flat, const float* dgate, const void* logits, const float* lse,
                                  const void* router, void* dlogits, void* dx, int tokens, int experts, int capacity, int d,
                                  mcclStream_t stream) {
  if (d < 0 || d % 8 || experts <= 0 || experts > kMaxExperts || !aligned16(dslots) || !aligned16(dx) || !aligned16(router)) return mcclInvalidArgument;
  if (tokens == 0) return mcclSuccess;
  const int smem = kRowWarps * experts * kTok * (int)sizeof(float);
  if (smem > 48 << 10 && cudaFuncSetAttribute(tokenBackwardKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return mcclSystemError;
  tokenBackwardKernel<<<rowBlocks((tokens + kTok - 1) / kTok), kRowThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(dslots), flat, dgate, static_cast<const __nv_bfloat16*>(logits), lse, static_cast<const uint4*>(router),
      tokens, experts, capacity, d / 8, static_cast<__nv_bfloat16*>(dlogits), static_cast<uint4*>(dx));
  return launchedOk();
}

}  // extern "C"
