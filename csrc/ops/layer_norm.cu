// LayerNorm and RMSNorm forward and backward for bf16 activations, rows of up to 4096 elements (a multiple of 8).
// A group of W warps owns a row, every lane holding VPL 16-byte vectors of it in registers, so a row is read once.
//   forward : mean / rstd by warp shuffles, y = (x - mean) * rstd * gamma + beta, mean and rstd saved in fp32.  With
//             `delta` the row is x + delta, rounded to bf16 and written out too: the residual add of a pre-norm block and
//             the norm behind it in one pass over memory.
//   backward: (rows of 256, 512 and 1024 elements of a LayerNorm have a kernel of their own, lnRowsBackwardKernel)
//             dx per row from two reductions; every lane also accumulates dgamma / dbeta of its columns over the rows its
//             group walks (col_reduce.cuh adds them up).  With `dres` the gradient that reaches the row past the norm (the
//             residual branch) is added (to the norm's gradient as a separate norm would have stored it), and the gradient
//             of y may come in up to three parts (one per projection that read y), added up here.  The column sums of the total can be had as well: the bias gradient of the
//             projection that produced `delta`.
// Both are bound by memory: forward 4 bytes an element (8 with delta), backward 6 (8 with dres).
// No counterpart in the reference (it has no model code).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "col_reduce.cuh"
#include "mccl.h"
#include "mccl_ops.h"

namespace {

using namespace mccl;

constexpr int kLnWarps = 8;
constexpr int kLnThreads = kLnWarps * 32;
constexpr int kLnMaxD = 4096;

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of (a, b) over the W warps of a row's group.  `slot`: shared memory of two floats a warp, alternating between two
// copies from call to call, which makes one barrier per call enough.
template <int W>
__device__ __forceinline__ float2 groupSum(float a, float b, float2* slot, int group, int warpInGroup) {
  a = warpSum(a); b = warpSum(b);
  if (W == 1) return make_float2(a, b);
  if ((threadIdx.x & 31) == 0) slot[group * W + warpInGroup] = make_float2(a, b);
  asm volatile("bar.sync %0, %1;" :: "r"(1 + group), "n"(W * 32) : "memory");
  float2 t = slot[group * W];
#pragma unroll
  for (int w = 1; w < W; ++w) { const float2 u = slot[group * W + w]; t.x += u.x; t.y += u.y; }
  return t;
}

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

// Sums of eight pairs, rounded as an addition of tensors rounds.
__device__ __forceinline__ uint4 add8(const uint4& a, const uint4& b) {
  float x[8], y[8];
  unpack(a, x);
  unpack(b, y);
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] += y[k];
  return pack(x);
}

// The arithmetic of a LayerNorm's gradient, its roundings spelled out: every form of the kernel gives the same bits.
__device__ __forceinline__ float normalised(float x, float mean, float rstd) { return __fmul_rn(__fsub_rn(x, mean), rstd); }
__device__ __forceinline__ float normGradient(float dy, float gamma, float xh, const float4& stats) {
  return __fmul_rn(stats.y, __fmaf_rn(-xh, stats.w, __fsub_rn(__fmul_rn(dy, gamma), stats.z)));
}

struct LnFwdArgs {
  const uint4 *x, *delta, *gamma, *beta;       // delta, beta: may be null
  uint4 *sum, *y;                              // sum: x + delta, written when delta is given
  float *mean, *rstd;                          // mean: null for RMSNorm
  int64_t rows;
  int D;
  float eps;
};

// One row per group and no loop: every load of a row is issued before the first wait, and 64 warps a SM keep up to 128 KB
// in flight.  Gamma and beta come from L1 after a CTA's first row.
template <int W, int VPL, bool RMS>
__global__ void __launch_bounds__(kLnThreads) lnForwardKernel(const __grid_constant__ LnFwdArgs a) {
  constexpr int G = kLnWarps / W, T = W * 32;
  __shared__ float2 slots[2][kLnWarps];
  const int group = threadIdx.x / T, t = threadIdx.x % T, vecs = a.D / 8;
  const int64_t row = (int64_t)blockIdx.x * G + group;
  if (row >= a.rows) return;
  const uint4* xr = a.x + row * vecs;
  const uint4* dr = a.delta + row * vecs;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 xq[VPL], dq[VPL], gq[VPL], bq[VPL];
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    const int i = t + T * j;
    const bool in = i < vecs;
    xq[j] = in ? xr[i] : zero;
    dq[j] = in && a.delta != nullptr ? dr[i] : zero;
    gq[j] = in ? a.gamma[i] : zero;
    bq[j] = in && !RMS ? a.beta[i] : zero;
  }
  float v[VPL * 8];
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    unpack(xq[j], v + 8 * j);
    if (a.delta != nullptr) {
      float d[8];
      unpack(dq[j], d);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[8 * j + k] += d[k];
      const uint4 q = pack(v + 8 * j);
      unpack(q, v + 8 * j);                    // the norm reads what a separate add would have stored
      if (t + T * j < vecs) a.sum[row * vecs + t + T * j] = q;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) { s += v[8 * j + k]; if (RMS) ss += v[8 * j + k] * v[8 * j + k]; }
  }
  const float invD = 1.0f / (float)a.D;
  float mu = 0.f, rs;
  if (RMS) {
    rs = rsqrtf(groupSum<W>(0.f, ss, slots[0], group, t >> 5).y * invD + a.eps);
  } else {
    mu = groupSum<W>(s, 0.f, slots[0], group, t >> 5).x * invD;
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < VPL; ++j)
      if (t + T * j < vecs)
#pragma unroll
        for (int k = 0; k < 8; ++k) { const float d = v[8 * j + k] - mu; sq += d * d; }
    rs = rsqrtf(groupSum<W>(sq, 0.f, slots[1], group, t >> 5).x * invD + a.eps);
  }
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    if (t + T * j >= vecs) continue;
    float g[8], b[8], y[8];
    unpack(gq[j], g);
    unpack(bq[j], b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (RMS) y[k] = __bfloat162float(__float2bfloat16_rn(v[8 * j + k] * rs)) * g[k];     // normalised, rounded, then scaled
      else y[k] = (v[8 * j + k] - mu) * rs * g[k] + b[k];
    }
    a.y[row * vecs + t + T * j] = pack(y);
  }
  if (t == 0) { if (!RMS) a.mean[row] = mu; a.rstd[row] = rs; }
}

struct LnBwdArgs {
  const uint4 *x, *dy, *dres, *gamma;          // dres: may be null
  const uint4 *dy2, *dy3;                      // more parts of dy, with PARTS == 3 (may be null there)
  const float *mean, *rstd;
  uint4* dx;
  float* partial;
  int64_t rows;
  int D;
  colred::Out out;                             // dgamma, dbeta, column sums of dx
};

// Sums of (a0, b0) and of (a1, b1) over the W warps of a group: four values through six exchanges, because every exchange
// also halves what a lane still carries, and one barrier.  `slot` as above, four floats a warp.
template <int W>
__device__ __forceinline__ float4 groupSum2(float a0, float b0, float a1, float b1, float4* slot, int group, int warpInGroup) {
  const int lane = threadIdx.x & 31;
  const bool second = lane & 16, isB = lane & 8;
  float a = (second ? a1 : a0) + __shfl_xor_sync(0xffffffffu, second ? a0 : a1, 16);
  float b = (second ? b1 : b0) + __shfl_xor_sync(0xffffffffu, second ? b0 : b1, 16);
  float v = (isB ? b : a) + __shfl_xor_sync(0xffffffffu, isB ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((lane & 7) == 0) reinterpret_cast<float*>(slot + group * W + warpInGroup)[lane >> 3] = v;
  asm volatile("bar.sync %0, %1;" :: "r"(1 + group), "n"(W * 32) : "memory");
  float4 t = slot[group * W];
#pragma unroll
  for (int w = 1; w < W; ++w) { const float4 u = slot[group * W + w]; t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w; }
  return t;
}

// Rows are walked by a fixed number of CTAs (two or three per SM) so that a lane can keep its columns' sums in registers; the
// vectors of the next rows are loaded before the current ones are worked on.  Two vectors per lane bound the registers: 16
// columns x (three sums + gamma) + two rows of x, dy and dres.
// R rows at a time.  What bounds the kernel is the chain of a row (the reductions' exchanges and the barrier between two
// passes over registers), so where a row is spread over warps and the registers suffice a group takes two rows and goes
// through the chain once for both (8192 x 1024 with dres: 21.4 us one row at a time, 18.4 us, 3.6 TB/s).  (A pipeline of four rows in shared memory by cp.async did not help: 25.9 us.)
template <int W, int VPL, bool RMS, bool RES, int PARTS, int R>
__global__ void __launch_bounds__(kLnThreads, VPL == 1 && PARTS == 1 && R == 1 ? 3 : 2) lnBackwardKernel(const __grid_constant__ LnBwdArgs a) {
  static_assert(R == 1 || (R == 2 && W > 1), "two rows at a time need a group of warps");
  constexpr int G = kLnWarps / W, T = W * 32;
  extern __shared__ float cols[];
  __shared__ float4 slots[2][kLnWarps];
  const int group = threadIdx.x / T, t = threadIdx.x % T, vecs = a.D / 8;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const bool third = RES && !RMS && a.out.segments == 3;
  float g[VPL * 8], dg[VPL * 8], db[VPL * 8], dc[VPL * 8];
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    unpack(t + T * j < vecs ? a.gamma[t + T * j] : zero, g + 8 * j);
#pragma unroll
    for (int k = 0; k < 8; ++k) dg[8 * j + k] = db[8 * j + k] = dc[8 * j + k] = 0.f;
  }
  const float invD = 1.0f / (float)a.D;
  const int64_t step = (int64_t)gridDim.x * (G * R);
  int64_t row = ((int64_t)blockIdx.x * G + group) * R;
  uint4 xq[R][VPL], dq[R][VPL], rq[R][VPL], d2[R][VPL], d3[R][VPL];
  float mu[R] = {}, rs[R] = {};
  auto load = [&](int64_t first) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int64_t r = first + q;
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        const int i = t + T * j;
        const bool in = r < a.rows && i < vecs;
        xq[q][j] = in ? a.x[r * vecs + i] : zero;
        dq[q][j] = in ? a.dy[r * vecs + i] : zero;
        if (RES) rq[q][j] = in ? a.dres[r * vecs + i] : zero;
        if (PARTS == 3) {
          d2[q][j] = in && a.dy2 != nullptr ? a.dy2[r * vecs + i] : zero;
          d3[q][j] = in && a.dy3 != nullptr ? a.dy3[r * vecs + i] : zero;
        }
      }
      const bool live = R == 1 || r < a.rows;                          // past the end everything is zero
      if (r < a.rows) { if (!RMS) mu[q] = a.mean[r]; rs[q] = a.rstd[r]; }
      if (!live) mu[q] = rs[q] = 0.f;
    }
  };
  load(row);
  for (int par = 0; row < a.rows; row += step, par ^= 1) {
    uint4 xc[R][VPL], dc4[R][VPL], rc[R][VPL];
    float m[R], r[R], s1[R], s2[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        xc[q][j] = xq[q][j];
        dc4[q][j] = PARTS == 3 ? add8(add8(dq[q][j], d2[q][j]), d3[q][j]) : dq[q][j];
        if (RES) rc[q][j] = rq[q][j];
      }
      m[q] = mu[q];
      r[q] = rs[q];
    }
    load(row + step);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      s1[q] = s2[q] = 0.f;
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        float xf[8], df[8];
        unpack(xc[q][j], xf);
        unpack(dc4[q][j], df);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float xh = (xf[k] - m[q]) * r[q], gd = df[k] * g[8 * j + k];
          s1[q] += gd; s2[q] += gd * xh;
          dg[8 * j + k] += df[k] * (RMS ? __bfloat162float(__float2bfloat16_rn(xh)) : xh);       // rows past the end: df is zero
          if (!RMS) db[8 * j + k] += df[k];
        }
      }
    }
    if (R == 2) {
      const float4 sums = groupSum2<W>(s1[0], s2[0], s1[R - 1], s2[R - 1], slots[par], group, t >> 5);
      s1[0] = sums.x; s2[0] = sums.y; s1[R - 1] = sums.z; s2[R - 1] = sums.w;
    } else {
      const float2 sums = groupSum<W>(s1[0], s2[0], reinterpret_cast<float2*>(slots[par]), group, t >> 5);
      s1[0] = sums.x; s2[0] = sums.y;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      if (R > 1 && row + q >= a.rows) continue;
      s1[q] = RMS ? 0.f : s1[q] * invD;
      s2[q] *= invD;
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        if (t + T * j >= vecs) continue;
        float xf[8], df[8], o[8];
        unpack(xc[q][j], xf);
        unpack(dc4[q][j], df);
        if (RES) unpack(rc[q][j], o);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float xh = (xf[k] - m[q]) * r[q], gd = df[k] * g[8 * j + k];
          const float dn = r[q] * (gd - s1[q] - xh * s2[q]);
          o[k] = RES ? __bfloat162float(__float2bfloat16_rn(dn)) + o[k] : dn;
        }
        const uint4 out = pack(o);
        if (third) {
          unpack(out, o);                      // the sum over what is stored, as a separate reduction would read it
#pragma unroll
          for (int k = 0; k < 8; ++k) dc[8 * j + k] += o[k];
        }
        a.dx[(row + q) * vecs + t + T * j] = out;
      }
    }
  }
  const int C = a.out.segments * a.D;
  float* mine = cols + group * C;
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    if (t + T * j >= vecs) continue;
    const int c = (t + T * j) * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      mine[c + k] = dg[8 * j + k];
      if (a.out.segments > 1) mine[a.D + c + k] = db[8 * j + k];
      if (third) mine[2 * a.D + c + k] = dc[8 * j + k];
    }
  }
  colred::finish(cols, G, C, a.partial, a.out);
}

// ---- LayerNorm backward for rows of 256, 512 and 1024 elements -----------------------------------------------------
// A batch of eight rows at a time.  A row's two sums need one order whatever else the kernel does (models are compared with
// runs of the separate operations, and one last bit here is a percent twenty layers down), so each warp takes one row of the
// batch for them: 32 lanes, VPL vectors each, one butterfly.  For the column sums that split is the wrong one (3 x 8 x VPL
// accumulators a lane), so the rows pass through shared memory and a thread then takes one vector of columns of VPL rows:
// 24 accumulators, and the gradients leave in whole rows.  One barrier a batch, because two copies of the rows alternate.
// 8192 x 1024 from cold caches: 23.6 us, 27.6 us with dres, 35.8 us with three parts, as long as the form below that spreads
// a row over four warps (and 29.7 us for one warp a row without the exchange, plain).
template <int VPL, bool RES, int PARTS>
__global__ void __launch_bounds__(kLnThreads, 2) lnRowsBackwardKernel(const __grid_constant__ LnBwdArgs a) {
  constexpr int VECS = VPL * 32, D = VPL * 256;
  extern __shared__ __align__(16) float cols[];
  uint4* sx = reinterpret_cast<uint4*>(cols);                          // [2][kLnWarps][VECS] rows of x, then as many of dy
  uint4* sd = sx + 2 * kLnWarps * VECS;
  __shared__ float4 stats[2][kLnWarps];                                // mean, rstd and the two sums of a row
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = threadIdx.x % VECS, slot0 = threadIdx.x / VECS * VPL;
  const bool third = RES && a.out.segments == 3;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  constexpr bool AHEAD = VPL * PARTS < 12;                             // the next batch's rows on their way: not with 24 vectors
  float g[8], dg[8], db[8], dc[8];
  unpack(a.gamma[c], g);
#pragma unroll
  for (int k = 0; k < 8; ++k) dg[k] = db[k] = dc[k] = 0.f;
  uint4 xq[VPL], dq[VPL], d2[VPL], d3[VPL];
  float mu = 0.f, rs = 0.f;
  auto load = [&](int64_t row) {
    const bool in = row < a.rows;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      const int64_t i = row * VECS + lane + 32 * j;
      xq[j] = in ? a.x[i] : zero;
      dq[j] = in ? a.dy[i] : zero;
      if (PARTS == 3) { d2[j] = in ? a.dy2[i] : zero; d3[j] = in ? a.dy3[i] : zero; }
    }
    if (in) { mu = a.mean[row]; rs = a.rstd[row]; }
  };
  const int64_t step = (int64_t)gridDim.x * kLnWarps;
  int64_t first = (int64_t)blockIdx.x * kLnWarps;
  if (AHEAD) load(first + warp);
  for (int par = 0; first < a.rows; first += step, par ^= 1) {
    if (!AHEAD) load(first + warp);
    float s1 = 0.f, s2 = 0.f;
    const int at = (par * kLnWarps + warp) * VECS + lane;
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
      float xf[8], df[8], gf[8];
      const uint4 dy = PARTS == 3 ? add8(add8(dq[j], d2[j]), d3[j]) : dq[j];
      sx[at + 32 * j] = xq[j];
      sd[at + 32 * j] = dy;
      unpack(xq[j], xf);
      unpack(dy, df);
      unpack(a.gamma[lane + 32 * j], gf);                              // from L1: sixteen registers a lane otherwise
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float gd = __fmul_rn(df[k], gf[k]);
        s1 = __fadd_rn(s1, gd);
        s2 = __fmaf_rn(gd, normalised(xf[k], mu, rs), s2);
      }
    }
    s1 = warpSum(s1) * (1.0f / D);
    s2 = warpSum(s2) * (1.0f / D);
    if (lane == 0) stats[par][warp] = make_float4(mu, rs, s1, s2);
    uint4 rq[VPL];
    if (RES) {
#pragma unroll
      for (int q = 0; q < VPL; ++q) rq[q] = first + slot0 + q < a.rows ? a.dres[(first + slot0 + q) * VECS + c] : zero;
    }
    if (AHEAD) load(first + step + warp);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < VPL; ++q) {
      const int slot = slot0 + q;
      if (first + slot >= a.rows) break;
      const float4 st = stats[par][slot];
      float xf[8], df[8], o[8];
      unpack(sx[(par * kLnWarps + slot) * VECS + c], xf);
      unpack(sd[(par * kLnWarps + slot) * VECS + c], df);
      if (RES) unpack(rq[q], o);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float xh = normalised(xf[k], st.x, st.y);
        const float dn = normGradient(df[k], g[k], xh, st);
        dg[k] += df[k] * xh;
        db[k] += df[k];
        o[k] = RES ? __bfloat162float(__float2bfloat16_rn(dn)) + o[k] : dn;
      }
      const uint4 out = pack(o);
      if (third) {
        unpack(out, o);                      // the sum over what is stored, as a separate reduction would read it
#pragma unroll
        for (int k = 0; k < 8; ++k) dc[k] += o[k];
      }
      a.dx[(first + slot) * VECS + c] = out;
    }
  }
  __syncthreads();                           // the rows' memory now takes the column sums
  float* mine = cols + threadIdx.x / VECS * (a.out.segments * D) + c * 8;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    mine[k] = dg[k];
    mine[D + k] = db[k];
    if (third) mine[2 * D + k] = dc[k];
  }
  colred::finish(cols, kLnWarps / VPL, a.out.segments * D, a.partial, a.out);
}

// ---- what is left of a LayerNorm's backward pass when the gradient through it is there (dn) -------------------------------
// dx = dn + dres and the column sums: dgamma, dbeta and those of dx.  One pass, a strip of 64 vectors of columns per CTA, four
// groups of 64 threads taking every fourth row, two rows in flight each.
constexpr int kTailVecs = 64, kTailGroups = kLnThreads / kTailVecs;

struct LnTailArgs {
  const uint4 *x, *dy, *dn, *dres;             // dres: may be null
  const float *mean, *rstd;
  uint4* dx;                                   // written where dres is given
  float* partial;
  int64_t rows;
  int D;
  colred::Out out;                             // dgamma, dbeta, column sums of dx
};

template <bool RES>
__global__ void __launch_bounds__(kLnThreads, 2) lnTailKernel(const __grid_constant__ LnTailArgs a) {
  __shared__ float red[colred::kMaxSegments][kTailGroups][kTailVecs * 8];
  const int tv = threadIdx.x % kTailVecs, group = threadIdx.x / kTailVecs, vecs = a.D / 8, v = blockIdx.x * kTailVecs + tv;
  float sum[colred::kMaxSegments][8] = {};
  if (v < vecs) {
    const int64_t step = (int64_t)gridDim.y * kTailGroups;
    for (int64_t r0 = (int64_t)blockIdx.y * kTailGroups + group; r0 < a.rows; r0 += 2 * step) {
      uint4 xq[2], dq[2], nq[2], rq[2];
      float mu[2], rs[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t r = r0 + u * step, i = r * vecs + v;
        if (r >= a.rows) continue;
        xq[u] = a.x[i];
        dq[u] = a.dy[i];
        nq[u] = a.dn[i];
        if (RES) rq[u] = a.dres[i];
        mu[u] = a.mean[r];
        rs[u] = a.rstd[r];
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t r = r0 + u * step;
        if (r >= a.rows) continue;
        float xf[8], df[8], o[8];
        unpack(xq[u], xf);
        unpack(dq[u], df);
        const uint4 dx = RES ? add8(nq[u], rq[u]) : nq[u];
        unpack(dx, o);
        if (RES) a.dx[r * vecs + v] = dx;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          sum[0][k] += df[k] * normalised(xf[k], mu[u], rs[u]);
          sum[1][k] += df[k];
          sum[2][k] += o[k];
        }
      }
    }
  }
#pragma unroll
  for (int s = 0; s < colred::kMaxSegments; ++s)
#pragma unroll
    for (int k = 0; k < 8; ++k) red[s][group][tv + kTailVecs * k] = sum[s][k];             // transposed: no bank conflicts
  __syncthreads();
  for (int i = threadIdx.x; i < a.out.segments * kTailVecs * 8; i += kLnThreads) {
    const int s = i / (kTailVecs * 8), c = i % (kTailVecs * 8), col = (blockIdx.x * kTailVecs + c % kTailVecs) * 8 + c / kTailVecs;
    if (col >= a.D) continue;
    float t = red[s][0][c];
#pragma unroll
    for (int g = 1; g < kTailGroups; ++g) t += red[s][g][c];
    if (gridDim.y == 1) colred::put(a.out, s * a.D + col, t);
    else a.partial[((int64_t)blockIdx.y * a.out.segments + s) * a.D + col] = t;
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <int W, int VPL, bool RMS>
cudaError_t fwd(const LnFwdArgs& a, cudaStream_t s) {
  constexpr int G = kLnWarps / W;
  lnForwardKernel<W, VPL, RMS><<<(unsigned)((a.rows + G - 1) / G), kLnThreads, 0, s>>>(a);
  return cudaGetLastError();
}

// Up to 1024 columns one warp holds a row (no barrier); wider rows are spread over four warps.
template <bool RMS>
cudaError_t fwdAny(const LnFwdArgs& a, cudaStream_t s) {
  if (a.D <= 256) return fwd<1, 1, RMS>(a, s);
  if (a.D <= 512) return fwd<1, 2, RMS>(a, s);
  if (a.D <= 768) return fwd<1, 3, RMS>(a, s);
  if (a.D <= 1024) return fwd<1, 4, RMS>(a, s);
  if (a.D <= 2048) return fwd<4, 2, RMS>(a, s);
  return fwd<4, 4, RMS>(a, s);
}

template <int W, int VPL, bool RMS, bool RES, int PARTS = 1, int R = 1>
cudaError_t bwdLaunch(const LnBwdArgs& a, cudaStream_t s) {
  constexpr int G = kLnWarps / W;
  const int C = a.out.segments * a.D, smem = G * C * (int)sizeof(float);
  if (smem > 40 << 10) {                       // with the row slots past the default limit; the same value from every thread and for every width
    const cudaError_t e = cudaFuncSetAttribute(lnBackwardKernel<W, VPL, RMS, RES, PARTS, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 << 10);
    if (e != cudaSuccess) return e;
  }
  int cluster;
  // Four rows a group, two turns where it takes two at a time: with four turns 512 x 1024 takes 15.4 us for 13.3, and more rows
  // the same.
  const int grid = colred::grid((a.rows + G * 4 - 1) / (G * 4), VPL == 1 && PARTS == 1 && R == 1 ? 3 : 2, &cluster);
  const cudaError_t e = colred::launch(lnBackwardKernel<W, VPL, RMS, RES, PARTS, R>, grid, cluster, kLnThreads, smem, s, a);
  return e != cudaSuccess ? e : colred::addPartials(a.partial, grid, cluster, C, a.out, s);
}

template <int VPL, bool RES, int PARTS>
cudaError_t bwdRows(const LnBwdArgs& a, cudaStream_t s) {
  constexpr int kRowBytes = 2 * kLnWarps * VPL * 512 * 2, kSumBytes = kLnWarps * 3 * 256 * (int)sizeof(float);
  constexpr int kSmem = kRowBytes > kSumBytes ? kRowBytes : kSumBytes;
  if (kSmem > 48 << 10) {
    const cudaError_t e = cudaFuncSetAttribute(lnRowsBackwardKernel<VPL, RES, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
  }
  int cluster;
  const int grid = colred::grid((a.rows + kLnWarps - 1) / kLnWarps, 2, &cluster);
  const cudaError_t e = colred::launch(lnRowsBackwardKernel<VPL, RES, PARTS>, grid, cluster, kLnThreads, kSmem, s, a);
  return e != cudaSuccess ? e : colred::addPartials(a.partial, grid, cluster, a.out.segments * a.D, a.out, s);
}
template <int VPL>
cudaError_t bwdRowsAny(const LnBwdArgs& a, cudaStream_t s) {
  if (!a.dres) return bwdRows<VPL, false, 1>(a, s);
  return a.dy2 ? bwdRows<VPL, true, 3>(a, s) : bwdRows<VPL, true, 1>(a, s);
}

// A lane's columns cost four registers each (three sums and gamma) beside two rows of x, dy and dres: two vectors a lane
// fit 128 registers without dres and spill with it (8192 x 1024: 26 us, with one vector a lane 19 us).
template <bool RMS, int PARTS>
cudaError_t bwdRes(const LnBwdArgs& a, cudaStream_t s) {
  if (a.D <= 256) return bwdLaunch<1, 1, RMS, true, PARTS>(a, s);
  constexpr int R = PARTS == 1 ? 2 : 1;        // five rows of operands leave no registers for a second one
  if (a.D <= 512) return bwdLaunch<2, 1, RMS, true, PARTS, R>(a, s);
  if (a.D <= 1024) return bwdLaunch<4, 1, RMS, true, PARTS, R>(a, s);
  if (a.D <= 2048) return bwdLaunch<8, 1, RMS, true, PARTS, R>(a, s);
  return bwdLaunch<8, 2, RMS, true, PARTS>(a, s);
}
template <bool RMS>
cudaError_t bwdAny(const LnBwdArgs& a, cudaStream_t s) {
  if (!RMS && a.D == 256) return bwdRowsAny<1>(a, s);
  if (!RMS && a.D == 512) return bwdRowsAny<2>(a, s);
  if (!RMS && a.D == 1024) return bwdRowsAny<4>(a, s);
  if (a.dres) return a.dy2 ? bwdRes<RMS, 3>(a, s) : bwdRes<RMS, 1>(a, s);
  if (a.D <= 256) return bwdLaunch<1, 1, RMS, false>(a, s);
  if (a.D <= 512) return bwdLaunch<1, 2, RMS, false>(a, s);
  if (a.D <= 1024) return bwdLaunch<2, 2, RMS, false>(a, s);
  if (a.D <= 2048) return bwdLaunch<4, 2, RMS, false>(a, s);
  return bwdLaunch<8, 2, RMS, false>(a, s);
}

mcclResult_t forward(const void* x, const void* delta, const void* gamma, const void* beta, void* sum, void* y, float* mean, float* rstd,
                     int64_t rows, int D, float eps, bool rms, mcclStream_t stream) {
  if (!x || !gamma || !y || !rstd || rows < 0 || (!rms && (!beta || !mean)) || (delta && !sum)) return mcclInvalidArgument;
  if (D <= 0 || D % 8 || D > kLnMaxD) return mcclInvalidArgument;
  if (!aligned16(x) || !aligned16(delta) || !aligned16(gamma) || !aligned16(beta) || !aligned16(sum) || !aligned16(y)) return mcclInvalidArgument;
  if (rows == 0) return mcclSuccess;
  LnFwdArgs a;
  a.x = static_cast<const uint4*>(x); a.delta = static_cast<const uint4*>(delta);
  a.gamma = static_cast<const uint4*>(gamma); a.beta = static_cast<const uint4*>(beta);
  a.sum = static_cast<uint4*>(sum); a.y = static_cast<uint4*>(y);
  a.mean = mean; a.rstd = rstd; a.rows = rows; a.D = D; a.eps = eps;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return (rms ? fwdAny<true>(a, s) : fwdAny<false>(a, s)) == cudaSuccess ? mcclSuccess : mcclSystemError;
}

mcclResult_t backward(const void* x, const void* dy, const void* dy2, const void* dy3, const void* dres, const void* gamma, const float* mean, const float* rstd, void* dx,
                      void* dgamma, void* dbeta, void* dcol, int accumulate, float* partial, int64_t rows, int D, bool rms,
                      mcclStream_t stream) {
  if (!x || !dy || !gamma || !rstd || !dx || !dgamma || !partial || rows <= 0 || (!rms && (!mean || !dbeta)) || (dcol && !dres) || (dy2 && !dres) || (dy3 && !dy2)) return mcclInvalidArgument;
  if (D <= 0 || D % 8 || D > kLnMaxD) return mcclInvalidArgument;
  if (!aligned16(x) || !aligned16(dy) || !aligned16(dres) || !aligned16(gamma) || !aligned16(dx) || !aligned16(dy2) || !aligned16(dy3)) return mcclInvalidArgument;
  LnBwdArgs a;
  a.dy2 = static_cast<const uint4*>(dy2); a.dy3 = static_cast<const uint4*>(dy3);
  a.x = static_cast<const uint4*>(x); a.dy = static_cast<const uint4*>(dy); a.dres = static_cast<const uint4*>(dres);
  a.gamma = static_cast<const uint4*>(gamma); a.mean = mean; a.rstd = rstd;
  a.dx = static_cast<uint4*>(dx); a.partial = partial; a.rows = rows; a.D = D;
  a.out = colred::Out{};
  a.out.seg[0] = static_cast<__nv_bfloat16*>(dgamma); a.out.seg[1] = static_cast<__nv_bfloat16*>(dbeta);
  a.out.seg[2] = static_cast<__nv_bfloat16*>(dcol);
  a.out.segments = dcol && dres ? 3 : dbeta ? 2 : 1; a.out.width = D; a.out.accumulate = accumulate;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return (rms ? bwdAny<true>(a, s) : bwdAny<false>(a, s)) == cudaSuccess ? mcclSuccess : mcclSystemError;
}

}  // namespace

// Partial sums the backward pass may write for `rows` rows (fp32, up to 3 x D each).
extern "C" int mcclLayerNormPartials(int64_t rows) { return rows <= 0 ? 1 : colred::kMaxPartials; }

extern "C" mcclResult_t mcclLayerNormForward(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                                             int64_t rows, int D, float eps, mcclStream_t stream) {
  return forward(x, nullptr, gamma, beta, nullptr, y, mean, rstd, rows, D, eps, false, stream);
}

// sum = x + delta (rounded to bf16), y = LayerNorm(sum).
extern "C" mcclResult_t mcclAddLayerNormForward(const void* x, const void* delta, const void* gamma, const void* beta, void* sum, void* y,
                                                float* mean, float* rstd, int64_t rows, int D, float eps, mcclStream_t stream) {
  if (!delta) return mcclInvalidArgument;
  return forward(x, delta, gamma, beta, sum, y, mean, rstd, rows, D, eps, false, stream);
}

// partial: fp32 work memory of mcclLayerNormPartials(rows) * 2 * D floats.
extern "C" mcclResult_t mcclLayerNormBackward(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd,
                                              void* dx, void* dgamma, void* dbeta, float* partial, int64_t rows, int D,
                                              mcclStream_t stream) {
  return backward(x, dy, nullptr, nullptr, nullptr, gamma, mean, rstd, dx, dgamma, dbeta, nullptr, 0, partial, rows, D, false, stream);
}

// The same with dx += dres and, when dcol is given, dcol = column sums of dx (needs dres); `accumulate`: add dgamma, dbeta and dcol to what
// is there.  dy2, dy3 (may be null, need dres): further parts of dy.  partial: mcclLayerNormPartials(rows) * 3 * D floats.
extern "C" mcclResult_t mcclAddLayerNormBackward(const void* x, const void* dy, const void* dy2, const void* dy3, const void* dres,
                                                 const void* gamma, const float* mean, const float* rstd, void* dx, void* dgamma, void* dbeta, void* dcol, int accumulate,
                                                 float* partial, int64_t rows, int D, mcclStream_t stream) {
  return backward(x, dy, dy2, dy3, dres, gamma, mean, rstd, dx, dgamma, dbeta, dcol, accumulate, partial, rows, D, false, stream);
}

// RMSNorm: y = bf16(x * rstd) * gamma; delta / sum as in mcclAddLayerNormForward (both may be null).
extern "C" mcclResult_t mcclRmsNormForward(const void* x, const void* delta, const void* gamma, void* sum, void* y, float* rstd,
                                           int64_t rows, int D, float eps, mcclStream_t stream) {
  return forward(x, delta, gamma, nullptr, sum, y, nullptr, rstd, rows, D, eps, true, stream);
}

extern "C" mcclResult_t mcclRmsNormBackward(const void* x, const void* dy, const void* dy2, const void* dy3, const void* dres, const void* gamma,
                                            const float* rstd, void* dx, void* dgamma, int accumulate, float* partial, int64_t rows, int D, mcclStream_t stream) {
  return backward(x, dy, dy2, dy3, dres, gamma, nullptr, rstd, dx, dgamma, nullptr, nullptr, accumulate, partial, rows, D, true, stream);
}

// The rest of a LayerNorm's backward pass with the gradient through it, dn, given: dx = dn + dres (dres and dx may be null: dx is
// dn), dgamma, dbeta and, when given, dcol = column sums of dx.  dy: the gradient of the norm's result.  partial as above.
extern "C" mcclResult_t mcclLayerNormBackwardTail(const void* x, const void* dy, const void* dn, const void* dres, const float* mean,
                                                  const float* rstd, void* dx, void* dgamma, void* dbeta, void* dcol, int accumulate,
                                                  float* partial, int64_t rows, int D, mcclStream_t stream) {
  if (!x || !dy || !dn || !mean || !rstd || !dgamma || !dbeta || !partial || rows <= 0 || D <= 0 || D % 8 || (dres && !dx)) return mcclInvalidArgument;
  if (!aligned16(x) || !aligned16(dy) || !aligned16(dn) || !aligned16(dres) || !aligned16(dx)) return mcclInvalidArgument;
  LnTailArgs a;
  a.x = static_cast<const uint4*>(x); a.dy = static_cast<const uint4*>(dy);
  a.dn = static_cast<const uint4*>(dn); a.dres = static_cast<const uint4*>(dres);
  a.mean = mean; a.rstd = rstd; a.dx = static_cast<uint4*>(dx); a.partial = partial; a.rows = rows; a.D = D;
  a.out = colred::Out{};
  a.out.seg[0] = static_cast<__nv_bfloat16*>(dgamma); a.out.seg[1] = static_cast<__nv_bfloat16*>(dbeta);
  a.out.seg[2] = static_cast<__nv_bfloat16*>(dcol);
  a.out.segments = dcol ? 3 : 2; a.out.width = D; a.out.accumulate = accumulate;
  // Two CTAs a SM, at least sixteen rows each.
  const int strips = (D / 8 + kTailVecs - 1) / kTailVecs;
  int64_t slices = 148 * 2 / strips;
  if (slices > (rows + 15) / 16) slices = (rows + 15) / 16;
  if (slices < 1) slices = 1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto* kernel = dres ? lnTailKernel<true> : lnTailKernel<false>;
  kernel<<<dim3(strips, (unsigned)slices), kLnThreads, 0, s>>>(a);
  if (cudaGetLastError() != cudaSuccess) return mcclSystemError;
  return colred::addPartials(partial, (int)slices, 1, a.out.segments * D, a.out, s) == cudaSuccess ? mcclSuccess : mcclSystemError;
}
