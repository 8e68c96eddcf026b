// Activations and their gradients over flat bf16 arrays: SiLU, SwiGLU and tanh-GELU, each one pass over memory with the
// arithmetic in fp32, and the GELU gradient together with its column sums (the bias gradient of the layer in front).
// Bound by memory: two to five 2-byte accesses an element.  Four 16-byte pieces of every operand are in flight per thread,
// which is what 6 TB/s takes at this occupancy; with one, the passes ran at half of that.
// No counterpart in the reference (it has no model code).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <initializer_list>

#include "col_reduce.cuh"
#include "f32x2.cuh"
#include "mccl.h"
#include "mccl_ops.h"

namespace {

using namespace mccl;

constexpr int kActThreads = 256;

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
// To fp32 precision, as the tensor library's: with __expf and __fdividef the gradients of SiLU round apart from 64 bits a little
// more often.
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }
// Of a bf16 number: rounded to bf16 the short form is the exact result for all of them below 80 (each was compared), in a
// good part less time (21 M elements 26.6 -> 22.5 us).
__device__ __forceinline__ float silu(float x) {
  return fabsf(x) < 80.f ? x * __fdividef(1.f, 1.f + __expf(-x)) : x / (1.f + expf(-x));
}

// The tanh-GELU is x * s with s = (1 + tanh(z)) / 2 = 1 / (1 + exp(-2 z)), z = c (x + a x^3): one exponential and one
// reciprocal, absolute error of s a few 2^-23, and its gradient is s + 2 z' x s (1 - s).  Results are to the last bit what the
// long form, with tanhf, rounds to: models are compared with runs of the separate operations, and one last bit here is a
// percent twenty layers down.  So the short form is only a guess with a bound: where both ends of its interval round to the
// same bf16 number that is the result, and elsewhere, about one value in a thousand, the long form decides.
constexpr float kGeluC = 0.7978845608028654f;      // sqrt(2 / pi)
constexpr float kGeluA = 0.044715f;
constexpr float kGeluGradW0 = 1.6e-7f, kGeluGradW2 = 1.3e-7f;
constexpr float kGeluE = -2.f * kGeluC * 1.4426950408889634f;      // exp(-2 z) = 2^(kGeluE (x + a x^3))
__device__ __forceinline__ float geluGate(float x, float x2) {
  float e, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * fmaf(kGeluE * kGeluA, x2, kGeluE)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.f + e));
  return s;
}

// Forward: the two forms differ by less than `w` (both within 3e-7 of 1 + tanh, products within 2^-22).
__device__ __noinline__ float geluLong(float x) {
  const float cube = x * x * x;
  return 0.5f * x * (1.f + tanhf(kGeluC * (x + kGeluA * cube)));
}
__device__ __forceinline__ uint32_t gelu2(float x0, float x1) {
  const float g0 = x0 * geluGate(x0, x0 * x0), g1 = x1 * geluGate(x1, x1 * x1);
  const float w0 = fmaf(fabsf(g0), 5e-7f, fabsf(x0) * 5e-7f), w1 = fmaf(fabsf(g1), 5e-7f, fabsf(x1) * 5e-7f);
  __nv_bfloat162 lo = __floats2bfloat162_rn(g0 - w0, g1 - w1), hi = __floats2bfloat162_rn(g0 + w0, g1 + w1);
  uint32_t a = *reinterpret_cast<uint32_t*>(&lo);
  const uint32_t b = *reinterpret_cast<uint32_t*>(&hi);
  if (a != b) {
    if ((a ^ b) & 0xffffu) lo.x = __float2bfloat16_rn(geluLong(x0));
    if ((a ^ b) >> 16) lo.y = __float2bfloat16_rn(geluLong(x1));
    a = *reinterpret_cast<uint32_t*>(&lo);
  }
  return a;
}

// Gradient of x from that of the result.  The two forms of gelu'(x) differ by less than `w` for |x| < 5.5 (at most by 2.1e-6,
// around |x| = 5, where the long form's 1 - t^2 cancels; all bf16 numbers were compared), and beyond that the long form is 1
// or 0.
constexpr uint32_t kGeluFlat = 0x40b0;             // 5.5 as bf16
__device__ __forceinline__ float geluGradLong(float x) {
  if (!(fabsf(x) < 5.5f)) return x > 0.f ? 1.f : x < 0.f ? 0.f : x;
  const float x2 = __fmul_rn(x, x), t = tanhf(__fmul_rn(kGeluC, __fmaf_rn(kGeluA, __fmul_rn(x2, x), x)));
  const float dz = __fmul_rn(kGeluC, __fmaf_rn(3.f * kGeluA, x2, 1.f));
  return __fadd_rn(__fmul_rn(0.5f, __fadd_rn(1.f, t)), __fmul_rn(__fmul_rn(__fmul_rn(0.5f, x), __fmaf_rn(-t, t, 1.f)), dz));
}
// The ends of the intervals of two products gelu'(x) dy, rounded.
__device__ __forceinline__ void geluGradEnds(uint32_t xw, uint32_t dyw, uint32_t* lo, uint32_t* hi) {
  const F2 x = f2OfBf16(xw), dy = f2OfBf16(dyw), x2 = x * x;
  float z0, z1, s0, s1;
  split(x * fma(f2(kGeluE * kGeluA), x2, f2(kGeluE)), &z0, &z1);
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(s0) : "f"(z0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(s1) : "f"(z1));
  split(f2(s0, s1) + f2(1.f), &z0, &z1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s0) : "f"(z0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s1) : "f"(z1));
  const F2 s = f2(s0, s1), g = fma(fma(s * f2(-1.f), s, s), x * fma(f2(6.f * kGeluC * kGeluA), x2, f2(2.f * kGeluC)), s);
  const F2 w = fma(f2(kGeluGradW2), x2, f2(kGeluGradW0));
  float a, b;
  split(dy * fma(w, f2(-1.f), g), &a, &b);
  __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
  *lo = *reinterpret_cast<uint32_t*>(&r);
  split(dy * (g + w), &a, &b);
  r = __floats2bfloat162_rn(a, b);
  *hi = *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t word(const uint4& q, int i) { return i & 2 ? (i & 1 ? q.w : q.z) : (i & 1 ? q.y : q.x); }
__device__ __forceinline__ float half(uint32_t w, int odd) { return __uint_as_float(odd ? w & 0xffff0000u : w << 16); }
// Eight gradients of x from eight of the result.
__device__ __forceinline__ uint4 geluGrad8(const uint4& x, const uint4& dy) {
  uint32_t o[4], open = 0;                                            // open: a bit for each that the long form decides
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t xw = word(x, j);
    uint32_t hi;
    geluGradEnds(xw, word(dy, j), &o[j], &hi);
    const uint32_t diff = o[j] ^ hi, flat = (xw & 0x7fff7fffu) + (0x8000u - kGeluFlat) * 0x10001u;     // bits 15 and 31: |x| >= 5.5 or NaN
    open |= (diff & 0xffffu ? 1u << (2 * j) : 0u) | (diff >> 16 ? 2u << (2 * j) : 0u);
    open |= (flat >> (15 - 2 * j) & 1u << (2 * j)) | (flat >> (30 - 2 * j) & 2u << (2 * j));
  }
  while (open != 0) {
    const int k = __ffs(open) - 1, j = k >> 1, odd = k & 1;
    open &= open - 1;
    const __nv_bfloat16 r = __float2bfloat16_rn(half(word(dy, j), odd) * geluGradLong(half(word(x, j), odd)));
    const uint32_t bits = __bfloat16_as_ushort(r);
#pragma unroll
    for (int i = 0; i < 4; ++i) if (i == j) o[i] = odd ? (o[i] & 0xffffu) | bits << 16 : (o[i] & 0xffff0000u) | bits;
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// An operation maps IN input values to OUT output values.
struct SiluFwd { static constexpr int IN = 1, OUT = 1; __device__ static void f(const float* i, float* o) { o[0] = silu(i[0]); } };
struct SiluBwd {                                   // (pre-activation, gradient) -> gradient of the pre-activation
  static constexpr int IN = 2, OUT = 1;
  __device__ static void f(const float* i, float* o) { const float s = sigmoid(i[0]); o[0] = i[1] * (s * (1.f + i[0] * (1.f - s))); }
};
struct SiluBoth {                                  // (pre-activation, gradient) -> activation, gradient of the pre-activation
  static constexpr int IN = 2, OUT = 2;
  __device__ static void f(const float* i, float* o) {
    const float s = sigmoid(i[0]);
    o[0] = i[0] * s;
    o[1] = i[1] * (s * (1.f + i[0] * (1.f - s)));
  }
};
struct SwigluFwd {                                 // (gate, up) -> silu(gate) * up, the activation rounded before the product
  static constexpr int IN = 2, OUT = 1;
  __device__ static void f(const float* i, float* o) { o[0] = rounded(silu(i[0])) * i[1]; }
};
struct SwigluBwd {                                 // (gate, up, gradient) -> product (for the weight gradient behind), d gate, d up
  static constexpr int IN = 3, OUT = 3;
  __device__ static void f(const float* i, float* o) {
    const float s = sigmoid(i[0]), act = rounded(i[0] * s);
    o[0] = act * i[1];
    o[1] = i[2] * i[1] * (s * (1.f + i[0] * (1.f - s)));
    o[2] = i[2] * act;
  }
};

template <class Op> struct ActArgs { const uint4* in[Op::IN]; uint4* out[Op::OUT]; int64_t n; };

template <class Op>
__global__ void __launch_bounds__(kActThreads) actKernel(const __grid_constant__ ActArgs<Op> a) {
  constexpr int U = Op::IN + Op::OUT >= 5 ? 2 : 4;
  const int64_t vecs = a.n / 8;
  const int64_t i0 = (int64_t)blockIdx.x * (kActThreads * U) + threadIdx.x;
  uint4 q[Op::IN][U];
#pragma unroll
  for (int k = 0; k < Op::IN; ++k)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * kActThreads < vecs) q[k][u] = a.in[k][i0 + u * kActThreads];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (i0 + u * kActThreads >= vecs) continue;
    float x[Op::IN][8], y[Op::OUT][8];
#pragma unroll
    for (int k = 0; k < Op::IN; ++k) unpack(q[k][u], x[k]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float in[Op::IN], out[Op::OUT];
#pragma unroll
      for (int k = 0; k < Op::IN; ++k) in[k] = x[k][e];
      Op::f(in, out);
#pragma unroll
      for (int k = 0; k < Op::OUT; ++k) y[k][e] = out[k];
    }
#pragma unroll
    for (int k = 0; k < Op::OUT; ++k) a.out[k][i0 + u * kActThreads] = pack(y[k]);
  }
  if (blockIdx.x == 0 && threadIdx.x < (unsigned)(a.n % 8)) {        // the last few elements
    const int64_t i = vecs * 8 + threadIdx.x;
    float in[Op::IN], out[Op::OUT];
#pragma unroll
    for (int k = 0; k < Op::IN; ++k) in[k] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.in[k])[i]);
    Op::f(in, out);
#pragma unroll
    for (int k = 0; k < Op::OUT; ++k) reinterpret_cast<__nv_bfloat16*>(a.out[k])[i] = __float2bfloat16_rn(out[k]);
  }
}

// GELU: four 16-byte pieces per thread as above; with the long form alone it was bound
// by arithmetic (8192 x 4096: 29.6 us; 26.2 us, 5.1 TB/s).
__global__ void __launch_bounds__(kActThreads) geluKernel(const uint4* x, uint4* y, int64_t n) {
  constexpr int U = 4;
  const int64_t vecs = n / 8, i0 = (int64_t)blockIdx.x * (kActThreads * U) + threadIdx.x;
  uint4 q[U];
#pragma unroll
  for (int u = 0; u < U; ++u) if (i0 + u * kActThreads < vecs) q[u] = x[i0 + u * kActThreads];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (i0 + u * kActThreads >= vecs) continue;
    float f[8];
    unpack(q[u], f);
    y[i0 + u * kActThreads] = make_uint4(gelu2(f[0], f[1]), gelu2(f[2], f[3]), gelu2(f[4], f[5]), gelu2(f[6], f[7]));
  }
  if (blockIdx.x == 0 && threadIdx.x < (unsigned)(n % 8)) {          // the last few elements
    const int64_t i = vecs * 8 + threadIdx.x;
    reinterpret_cast<__nv_bfloat16*>(y)[i] = __float2bfloat16_rn(geluLong(__bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i])));
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <class Op>
mcclResult_t act(std::initializer_list<const void*> in, std::initializer_list<void*> out, int64_t n, mcclStream_t stream) {
  ActArgs<Op> a;
  int k = 0;
  for (const void* p : in) { if (p == nullptr || !aligned16(p)) return mcclInvalidArgument; a.in[k++] = static_cast<const uint4*>(p); }
  k = 0;
  for (void* p : out) { if (p == nullptr || !aligned16(p)) return mcclInvalidArgument; a.out[k++] = static_cast<uint4*>(p); }
  if (n < 0) return mcclInvalidArgument;
  if (n == 0) return mcclSuccess;
  a.n = n;
  constexpr int U = Op::IN + Op::OUT >= 5 ? 2 : 4;
  const int64_t per = (int64_t)kActThreads * U, blocks = (n / 8 + per - 1) / per;
  actKernel<Op><<<(unsigned)(blocks < 1 ? 1 : blocks), kActThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

// ---- column sums ------------------------------------------------------------------------------------------------------
// A CTA takes a strip of 64 x 8 columns (one vector per lane of two warps' width) and walks rows; four groups of 64 threads
// take every fourth row.  Up to three matrices of the same shape in one launch (blockIdx.z).  With GELU the matrix is the
// gradient of the activation, replaced by the gradient of the pre-activation on the way (8192 x 4096: 44.9 us, 4.5 TB/s, of
// which the last bits of the long form are 6 us).  With PACK the matrices are also written side by side into one
// [rows, segments x D] matrix, so that the product behind takes them as one operand: for 8192 tokens and width 1024 three weight
// gradients of 1024 x 1024 (77 us, too small to fill the GPU with large tiles) become one product (35 us), and this pass goes
// from 9.5 to 14.0 us.
enum ColMode { COL_SUM, COL_GELU, COL_PACK };
constexpr int kStripVecs = 64, kStripCols = kStripVecs * 8, kRowGroups = kActThreads / kStripVecs;

struct ColArgs {
  const uint4* x[colred::kMaxSegments];       // [rows, D] each, row stride `ld` vectors
  const uint4* pre;                           // GELU: pre-activation
  uint4* dx;                                  // GELU: where the gradient goes; PACK: the matrix of all
  float* partial;                             // [gridDim.y][segments * D]
  int64_t rows, ld, ldx;                      // ldx: row stride of dx
  int D;
  colred::Out out;
};

template <int MODE>
__global__ void __launch_bounds__(kActThreads, 3) colSumKernel(const __grid_constant__ ColArgs a) {
  constexpr bool GELU = MODE == COL_GELU;
  __shared__ float red[kRowGroups][kStripCols];
  const int tv = threadIdx.x % kStripVecs, g = threadIdx.x / kStripVecs, vecs = a.D / 8;
  const int v = blockIdx.x * kStripVecs + tv, seg = blockIdx.z;
  // Rows in flight per thread.  The GELU's arithmetic takes as long as its loads, so there the next rows are on their way
  // meanwhile.
  constexpr int U = GELU ? 2 : 4;
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (v < vecs) {
    const uint4* x = a.x[seg];
    const int64_t step = (int64_t)gridDim.y * kRowGroups;
    uint4 q[U], p[U], qn[U], pn[U];
    auto load = [&](int64_t first, uint4* to, uint4* pre) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t r = first + u * step;
        if (r < a.rows) { to[u] = x[r * a.ld + v]; if (GELU) pre[u] = a.pre[r * a.ld + v]; }
      }
    };
    int64_t r0 = (int64_t)blockIdx.y * kRowGroups + g;
    if (GELU) load(r0, qn, pn);
    for (; r0 < a.rows; r0 += U * step) {
      if (GELU) {
#pragma unroll
        for (int u = 0; u < U; ++u) { q[u] = qn[u]; p[u] = pn[u]; }
        load(r0 + U * step, qn, pn);
      } else {
        load(r0, q, p);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t r = r0 + u * step;
        if (r >= a.rows) continue;
        uint4 o = q[u];
        if (GELU) o = geluGrad8(p[u], q[u]);
        if (GELU) a.dx[r * a.ldx + v] = o;
        if (MODE == COL_PACK) a.dx[r * a.ldx + (int64_t)seg * vecs + v] = o;
        float f[8];
        unpack(o, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) sum[k] += f[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) red[g][tv + kStripVecs * k] = sum[k];      // transposed: no bank conflicts
  __syncthreads();
  for (int c = threadIdx.x; c < kStripCols; c += kActThreads) {
    float t = red[0][c];
#pragma unroll
    for (int i = 1; i < kRowGroups; ++i) t += red[i][c];
    const int col = (blockIdx.x * kStripVecs + c % kStripVecs) * 8 + c / kStripVecs;
    if (col >= a.D) continue;
    if (gridDim.y == 1) colred::put(a.out, seg * a.D + col, t);
    else a.partial[((int64_t)blockIdx.y * gridDim.z + seg) * a.D + col] = t;
  }
}

// Row slices: enough CTAs for three per SM, at least 16 rows a slice (four rows in flight for each of the four row groups).
int colSlices(int64_t rows, int D, int segments) {
  const int64_t strips = (int64_t)((D / 8 + kStripVecs - 1) / kStripVecs) * segments;
  int64_t s = 148 * 3 / strips;
  const int64_t most = (rows + 15) / 16;
  if (s > most) s = most;
  if (s > colred::kMaxPartials) s = colred::kMaxPartials;
  return s < 1 ? 1 : (int)s;
}

template <int MODE>
mcclResult_t colSums(const ColArgs& a, cudaStream_t s) {
  const int strips = (a.D / 8 + kStripVecs - 1) / kStripVecs, slices = colSlices(a.rows, a.D, a.out.segments);
  colSumKernel<MODE><<<dim3(strips, slices, a.out.segments), kActThreads, 0, s>>>(a);
  if (cudaGetLastError() != cudaSuccess) return mcclSystemError;
  return colred::addPartials(a.partial, slices, 1, a.out.segments * a.D, a.out, s) == cudaSuccess ? mcclSuccess : mcclSystemError;
}

}  // namespace

extern "C" mcclResult_t mcclSiluForward(const void* x, void* y, int64_t n, mcclStream_t s) { return act<SiluFwd>({x}, {y}, n, s); }
extern "C" mcclResult_t mcclSiluBackward(const void* x, const void* dy, void* dx, int64_t n, mcclStream_t s) { return act<SiluBwd>({x, dy}, {dx}, n, s); }
extern "C" mcclResult_t mcclSiluForwardBackward(const void* x, const void* dy, void* y, void* dx, int64_t n, mcclStream_t s) {
  return act<SiluBoth>({x, dy}, {y, dx}, n, s);
}
extern "C" mcclResult_t mcclSwigluForward(const void* gate, const void* up, void* y, int64_t n, mcclStream_t s) { return act<SwigluFwd>({gate, up}, {y}, n, s); }
extern "C" mcclResult_t mcclSwigluBackward(const void* gate, const void* up, const void* dy, void* y, void* dgate, void* dup, int64_t n, mcclStream_t s) {
  return act<SwigluBwd>({gate, up, dy}, {y, dgate, dup}, n, s);
}
extern "C" mcclResult_t mcclGeluForward(const void* x, void* y, int64_t n, mcclStream_t stream) {
  if (!x || !y || !aligned16(x) || !aligned16(y) || n < 0) return mcclInvalidArgument;
  if (n == 0) return mcclSuccess;
  const int64_t per = kActThreads * 4, blocks = (n / 8 + per - 1) / per;
  geluKernel<<<(unsigned)(blocks < 1 ? 1 : blocks), kActThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), static_cast<uint4*>(y), n);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

// Floats of work memory the two functions below need.
extern "C" int64_t mcclColumnSumScratch(int64_t rows, int D, int segments) {
  return rows <= 0 || D <= 0 || segments <= 0 ? 0 : (int64_t)colSlices(rows, D, segments) * segments * D;
}

// dx = dy * gelu'(x) for [rows, D] matrices, dbias (nullable) = [+] column sums of dx.
extern "C" mcclResult_t mcclGeluBackward(const void* x, const void* dy, void* dx, void* dbias, int accumulate, float* scratch, int64_t rows,
                                         int D, mcclStream_t stream) {
  if (!x || !dy || !dx || !scratch || rows <= 0 || D <= 0 || D % 8 || !aligned16(x) || !aligned16(dy) || !aligned16(dx)) return mcclInvalidArgument;
  ColArgs a = {};
  a.x[0] = static_cast<const uint4*>(dy); a.pre = static_cast<const uint4*>(x); a.dx = static_cast<uint4*>(dx);
  a.partial = scratch; a.rows = rows; a.ld = a.ldx = D / 8; a.D = D;
  a.out.seg[0] = static_cast<__nv_bfloat16*>(dbias); a.out.segments = 1; a.out.width = D; a.out.accumulate = accumulate;
  return colSums<COL_GELU>(a, reinterpret_cast<cudaStream_t>(stream));
}

// out[i] = [+] column sums of x[i], up to three [rows, D] matrices with rows `ld` elements apart.
extern "C" mcclResult_t mcclColumnSums(const void* const* x, void* const* out, int n, int accumulate, float* scratch, int64_t rows, int D,
                                       int64_t ld, mcclStream_t stream) {
  if (!x || !out || !scratch || n < 1 || n > colred::kMaxSegments || rows <= 0 || D <= 0 || D % 8 || ld < D || ld % 8) return mcclInvalidArgument;
  ColArgs a = {};
  for (int i = 0; i < n; ++i) {
    if (!x[i] || !out[i] || !aligned16(x[i])) return mcclInvalidArgument;
    a.x[i] = static_cast<const uint4*>(x[i]);
    a.out.seg[i] = static_cast<__nv_bfloat16*>(out[i]);
  }
  a.partial = scratch; a.rows = rows; a.ld = ld / 8; a.D = D;
  a.out.segments = n; a.out.width = D; a.out.accumulate = accumulate;
  return colSums<COL_SUM>(a, reinterpret_cast<cudaStream_t>(stream));
}

// The same for contiguous matrices, which are also written side by side: packed[r][i * D + c] = x[i][r][c].
extern "C" mcclResult_t mcclPackColumnSums(const void* const* x, void* packed, void* const* out, int n, int accumulate, float* scratch,
                                           int64_t rows, int D, mcclStream_t stream) {
  if (!x || !packed || !out || !scratch || n < 1 || n > colred::kMaxSegments || rows <= 0 || D <= 0 || D % 8 || !aligned16(packed))
    return mcclInvalidArgument;
  ColArgs a = {};
  for (int i = 0; i < n; ++i) {
    if (!x[i] || !out[i] || !aligned16(x[i])) return mcclInvalidArgument;
    a.x[i] = static_cast<const uint4*>(x[i]);
    a.out.seg[i] = static_cast<__nv_bfloat16*>(out[i]);
  }
  a.dx = static_cast<uint4*>(packed);
  a.partial = scratch; a.rows = rows; a.ld = D / 8; a.ldx = (int64_t)n * (D / 8); a.D = D;
  a.out.segments = n; a.out.width = D; a.out.accumulate = accumulate;
  return colSums<COL_PACK>(a, reinterpret_cast<cudaStream_t>(stream));
}
