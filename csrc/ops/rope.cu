// Rotary position embedding of q and k in one pass: a thread turns eight pairs (i, i + hd/2) of several heads, so the angles of
// its token and pairs are worked out once, in fp32, and used for all of them.  Bound by memory (4 bytes an element); as
// separate fp32 tensor operations it was a dozen passes, 16 to 24 bytes an element each.
// No counterpart in the reference (it has no model code).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mccl.h"
#include "mccl_ops.h"

namespace {

constexpr int kRopeThreads = 128;
constexpr int kRopeHeads = 4;                  // heads per thread

struct RopeArgs {
  const __nv_bfloat16* src[2];
  __nv_bfloat16* dst[2];
  int64_t tokens, sb, ss, sh;
  int seq, heads, hd;
  float theta;
  int inverse;
};

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

// grid: (tokens x pieces of eight pairs, groups of heads, arrays)
__global__ void __launch_bounds__(kRopeThreads) ropeKernel(const __grid_constant__ RopeArgs a) {
  const int half = a.hd / 2, pieces = half / 8;
  const int64_t i = (int64_t)blockIdx.x * kRopeThreads + threadIdx.x;
  if (i >= a.tokens * pieces) return;
  const int64_t t = i / pieces, b = t / a.seq;
  const int p = (int)(i - t * pieces), s = (int)(t - b * a.seq), h0 = blockIdx.y * kRopeHeads;
  const __nv_bfloat16* src = a.src[blockIdx.z] + b * a.sb + (int64_t)s * a.ss + p * 8;
  __nv_bfloat16* dst = a.dst[blockIdx.z] + t * ((int64_t)a.heads * a.hd) + p * 8;
  uint4 lo[kRopeHeads], hi[kRopeHeads];
#pragma unroll
  for (int h = 0; h < kRopeHeads; ++h) {
    if (h0 + h >= a.heads) continue;
    const __nv_bfloat16* x = src + (int64_t)(h0 + h) * a.sh;
    lo[h] = *reinterpret_cast<const uint4*>(x);
    hi[h] = *reinterpret_cast<const uint4*>(x + half);
  }
  float c[8], sn[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float freq = powf(a.theta, -(float)(p * 8 + k) / (float)half);
    sincosf((float)s * freq, &sn[k], &c[k]);
    if (a.inverse) sn[k] = -sn[k];
  }
#pragma unroll
  for (int h = 0; h < kRopeHeads; ++h) {
    if (h0 + h >= a.heads) continue;
    float x[8], y[8], u[8], v[8];
    unpack(lo[h], x);
    unpack(hi[h], y);
#pragma unroll
    for (int k = 0; k < 8; ++k) { u[k] = x[k] * c[k] - y[k] * sn[k]; v[k] = x[k] * sn[k] + y[k] * c[k]; }
    __nv_bfloat16* o = dst + (int64_t)(h0 + h) * a.hd;
    *reinterpret_cast<uint4*>(o) = pack(u);
    *reinterpret_cast<uint4*>(o + half) = pack(v);
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

extern "C" mcclResult_t mcclRope(const void* src0, const void* src1, void* dst0, void* dst1, int batch, int seq, int heads, int hd, int64_t sb,
                                 int64_t ss, int64_t sh, float theta, int inverse, mcclStream_t stream) {
  if (!src0 || !dst0 || !src1 != !dst1 || batch <= 0 || seq <= 0 || heads <= 0 || hd <= 0 || hd % 16 || sb % 8 || ss % 8 || sh % 8) return mcclInvalidArgument;
  if (!aligned16(src0) || !aligned16(src1) || !aligned16(dst0) || !aligned16(dst1)) return mcclInvalidArgument;
  RopeArgs a;
  a.src[0] = static_cast<const __nv_bfloat16*>(src0); a.src[1] = static_cast<const __nv_bfloat16*>(src1);
  a.dst[0] = static_cast<__nv_bfloat16*>(dst0); a.dst[1] = static_cast<__nv_bfloat16*>(dst1);
  a.tokens = (int64_t)batch * seq; a.sb = sb; a.ss = ss; a.sh = sh; a.seq = seq; a.heads = heads; a.hd = hd; a.theta = theta; a.inverse = inverse;
  const int64_t n = a.tokens * (hd / 16);
  ropeKernel<<<dim3((unsigned)((n + kRopeThreads - 1) / kRopeThreads), (heads + kRopeHeads - 1) / kRopeHeads, src1 ? 2 : 1), kRopeThreads, 0,
               reinterpret_cast<cudaStream_t>(stream)>>>(a);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}
