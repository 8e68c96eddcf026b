// Sum of squares of a bf16 array (the global gradient norm of a training step, accumulated bucket by
// bucket).  Two stages inside one launch: every block folds one fixed tile into a partial sum in scratch
// memory; the block that finishes last (a ticket counter, also in scratch) adds the partials in index
// order, so the result does not depend on which block finished when.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace mccl {

constexpr int kNormThreads = 256;
constexpr uint64_t kNormTile = 65536;          // elements per block, at most
constexpr uint64_t kNormTileSmall = 16384;     // ... of arrays that this tile cuts into 4096 blocks or fewer
constexpr int kNormUnroll = 8;                 // 16-byte pieces in flight per thread: the whole of a small tile
constexpr uint64_t kNormHeader = 64;           // floats reserved in front of the partials (ticket counter)

// Bound by memory (2 bytes an element).  The small tile gives a 25 MB bucket 800 blocks instead of 200, so the last wave
// is not nearly empty, and each thread has its whole share in flight: 10.5 us -> 7.7 us.
inline uint64_t normTile(uint64_t n) { return n <= 4096 * kNormTileSmall ? kNormTileSmall : kNormTile; }

// scratch layout: [0] ticket counter (as unsigned), [kNormHeader ...) one partial per block.
static __global__ void __launch_bounds__(kNormThreads) sumSquaresKernel(const __nv_bfloat16* x, uint64_t n, float* scratch,
                                                                 float* out, int accumulate, uint64_t tile) {
  __shared__ float warpSums[kNormThreads / 32];
  __shared__ unsigned ticket;
  const uint64_t lo = (uint64_t)blockIdx.x * tile;
  const uint64_t hi = lo + tile < n ? lo + tile : n;
  float acc = 0.f;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  if (vec) {
    const uint64_t v0 = lo / 8, v1 = hi / 8;                 // lo is a multiple of the tile, hence of 8
    for (uint64_t i = v0 + threadIdx.x; i < v1; i += kNormUnroll * kNormThreads) {
      uint4 q[kNormUnroll];
#pragma unroll
      for (int u = 0; u < kNormUnroll; ++u) {
        const uint64_t k = i + (uint64_t)u * kNormThreads;
        q[u] = k < v1 ? reinterpret_cast<const uint4*>(x)[k] : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < kNormUnroll; ++u) {
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&q[u]);
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float2 f = __bfloat1622float2(e[k]); acc += f.x * f.x; acc += f.y * f.y; }
      }
    }
    for (uint64_t i = v1 * 8 + threadIdx.x; i < hi; i += kNormThreads) { const float f = __bfloat162float(x[i]); acc += f * f; }
  } else {
    for (uint64_t i = lo + threadIdx.x; i < hi; i += kNormThreads) { const float f = __bfloat162float(x[i]); acc += f * f; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) warpSums[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < kNormThreads / 32; ++w) s += warpSums[w];
    scratch[kNormHeader + blockIdx.x] = s;
    __threadfence();
    ticket = atomicAdd(reinterpret_cast<unsigned*>(scratch), 1u);
  }
  __syncthreads();
  if (ticket != gridDim.x - 1) return;
  // Last block: every partial is visible (each writer fenced before taking its ticket).
  __threadfence();
  float s = 0.f;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += kNormUnroll * kNormThreads) {
    float p[kNormUnroll];
#pragma unroll
    for (int u = 0; u < kNormUnroll; ++u) p[u] = i + u * kNormThreads < gridDim.x ? __ldcg(scratch + kNormHeader + i + u * kNormThreads) : 0.f;
#pragma unroll
    for (int u = 0; u < kNormUnroll; ++u) s += p[u];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) warpSums[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < kNormThreads / 32; ++w) t += warpSums[w];
    *out = accumulate ? *out + t : t;
    *reinterpret_cast<unsigned*>(scratch) = 0u;            // ready for the next launch
  }
}

inline uint64_t normBlocks(uint64_t n) { const uint64_t t = normTile(n); return (n + t - 1) / t; }

}  // namespace mccl
