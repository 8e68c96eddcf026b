// Sums over rows, one per column (the gradients of biases and norm weights), as the tail of kernels that walk the rows
// anyway, all in a fixed order: a CTA folds its row groups in shared memory, and a small second kernel adds the CTAs' sums
// (296 partials of 2048 columns: 2.5 us).  Inputs that need eight CTAs or fewer run as one cluster, whose CTAs fold through
// distributed shared memory and write the result: one launch.  (Clusters of four for the large grid too would shorten the
// second kernel, but 74 such clusters do not fit the SMs of the GPCs at once: the first kernel took two waves, 45 us for 20.)
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mccl {
namespace colred {

constexpr int kMaxSegments = 3;
constexpr int kMaxCtas = 444;                 // three CTAs per SM
constexpr int kMaxPartials = kMaxCtas;

// Where the sums of columns [i * width, (i + 1) * width) go (null: nowhere), as bf16.
struct Out {
  __nv_bfloat16* seg[kMaxSegments];
  int segments;
  int width;
  int accumulate;                             // add to what is there (a gradient buffer) instead of overwriting it
};

__device__ __forceinline__ void put(const Out& o, int c, float t) {
  const int s = c / o.width, k = c - s * o.width;
  __nv_bfloat16* p = o.seg[s];
  if (p == nullptr) return;
  p[k] = __float2bfloat16_rn(o.accumulate ? __bfloat162float(p[k]) + t : t);
}

__device__ __forceinline__ uint32_t clusterRank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t clusterSize() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void clusterSync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float ldPeerShared(const float* local, uint32_t cta) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(local), r;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
  return v;
}

// `cols`: this CTA's `groups` arrays of `C` column sums, in shared memory and written by all threads before the call.
// Every thread of every CTA calls this once, last.  C = o.segments * o.width.
__device__ __forceinline__ void finish(float* cols, int groups, int C, float* partial, const Out& o) {
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float t = cols[c];
    for (int g = 1; g < groups; ++g) t += cols[g * C + c];
    cols[c] = t;
  }
  const uint32_t R = clusterSize(), r = clusterRank();
  if (R > 1) clusterSync(); else __syncthreads();
  const int lo = (int)((int64_t)C * r / R), hi = (int)((int64_t)C * (r + 1) / R);
  const bool whole = gridDim.x == R;
  float* mine = partial + (int64_t)(blockIdx.x / R) * C;
  for (int c = lo + threadIdx.x; c < hi; c += blockDim.x) {
    float t = 0.f;
    for (uint32_t p = 0; p < R; ++p) t += ldPeerShared(cols + c, p);
    if (whole) put(o, c, t); else mine[c] = t;
  }
  if (R > 1) clusterSync();                   // nobody leaves while a peer still reads its shared memory
}

// 32 columns per CTA, 32 warps: up to 444 partials are fourteen loads per thread, all in flight together.
static __global__ void __launch_bounds__(1024) addPartialsKernel(const float* partial, int P, int C, const __grid_constant__ Out o) {
  __shared__ float acc[32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  constexpr int U = (kMaxPartials + 31) / 32;
  float x[U], t = 0.f;
#pragma unroll
  for (int i = 0; i < U; ++i) { const int p = warp + 32 * i; x[i] = p < P && c < C ? partial[(int64_t)p * C + c] : 0.f; }
#pragma unroll
  for (int i = 0; i < U; ++i) t += x[i];
  acc[warp][lane] = t;
  __syncthreads();
  float v = acc[lane][warp];                  // warp w adds column w of the 32 x 32 tile
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) v += __shfl_xor_sync(0xffffffffu, v, k);
  const int cc = blockIdx.x * 32 + warp;
  if (lane == 0 && cc < C) put(o, cc, v);
}

// CTAs for `items` units of work (one unit: what a CTA does between two looks at its loop condition), *cluster = CTAs per cluster.
inline int grid(int64_t items, int perSm, int* cluster) {
  if (items <= 8) { *cluster = items < 1 ? 1 : (int)items; return *cluster; }
  *cluster = 1;
  return items > 148 * perSm ? 148 * perSm : (int)items;
}

template <typename... Params, typename... Args>
inline cudaError_t launch(void (*kernel)(Params...), int grid, int cluster, int threads, int smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// The second level, where there is one.
inline cudaError_t addPartials(const float* partial, int grid, int cluster, int C, const Out& o, cudaStream_t s) {
  if (grid == cluster) return cudaSuccess;
  addPartialsKernel<<<(C + 31) / 32, 1024, 0, s>>>(partial, grid / cluster, C, o);
  return cudaGetLastError();
}

}  // namespace colred
}  // namespace mccl
