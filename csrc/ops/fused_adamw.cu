// Fused AdamW over one flat gradient bucket: reads the (already averaged) bf16 gradients in place in the
// bucket the all-reduce wrote, updates fp32 master weights and both moments, and writes the bf16 working
// copy of the parameters: one pass over memory instead of the dozen elementwise kernels of an unfused step.
// Exposed through the C ABI so the Python side can call it with raw pointers on any stream.
// No counterpart in the reference (it has no training code); this is the optimizer half of the
// data-parallel step its benchmark describes (docs/perf-scaling.png: "compute on batch + gradient all-reduce").
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mccl.h"
#include "mccl_ops.h"

namespace {

struct AdamArgs {
  __nv_bfloat16* param;      // bf16 working weights (what the model reads)
  float* master;             // fp32 master weights
  float* expAvg;
  float* expAvgSq;
  const __nv_bfloat16* grad; // bf16 gradients (bucket)
  uint64_t n;
  float lr, beta1, beta2, eps, weightDecay, gradScale, biasCorr1, biasCorr2Sqrt;
  int zeroGrad;              // clear the gradient after use, ready for the next accumulation
  const float* normSq;       // optional device scalar: squared global gradient norm (for clipping)
  float maxNorm;             // clip threshold; used only when normSq is set
  const float* hyper;        // optional device array {lr, 1 - beta1^t, sqrt(1 - beta2^t)}: read at run time, so a
                             // launch recorded in a CUDA graph follows the schedule when it is replayed
};

// Eight floats with one access: a lane's 32 bytes are a whole sector, where two 16-byte stores leave the L2 with two
// partial writes of it.  WIDE needs 32-byte aligned arrays.
template <bool WIDE> __device__ __forceinline__ void ld8(const float* p, float* f) {
  if (WIDE) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]),
                 "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(p) : "memory");
  } else {
    const float4 x = reinterpret_cast<const float4*>(p)[0], y = reinterpret_cast<const float4*>(p)[1];
    f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w; f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
  }
}
template <bool WIDE> __device__ __forceinline__ void st8(float* p, const float* f) {
  if (WIDE) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" :: "l"(p), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]),
                 "f"(f[5]), "f"(f[6]), "f"(f[7]) : "memory");
  } else {
    reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(256) adamwKernel(const __grid_constant__ AdamArgs arg) {
  AdamArgs a = arg;
  if (a.hyper != nullptr) { a.lr = a.hyper[0]; a.biasCorr1 = a.hyper[1]; a.biasCorr2Sqrt = a.hyper[2]; }
  if (a.normSq != nullptr) {   // global-norm clipping: scale = min(1, maxNorm / ||g||), read on the device (no host sync)
    const float norm = sqrtf(*a.normSq) * a.gradScale;
    if (norm > a.maxNorm) a.gradScale *= a.maxNorm / (norm + 1e-6f);
  }
  const uint64_t nVec = a.n / 8;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = tid; i < nVec; i += nth) {
    uint4 gq = reinterpret_cast<const uint4*>(a.grad)[i];
    const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(&gq);
    float wf[8], mf[8], vf[8];
    ld8<WIDE>(a.master + 8 * i, wf);
    ld8<WIDE>(a.expAvg + 8 * i, mf);
    ld8<WIDE>(a.expAvgSq + 8 * i, vf);
    uint4 pq;
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(&pq);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float gr = __bfloat162float(g[k]) * a.gradScale;
      mf[k] = a.beta1 * mf[k] + (1.f - a.beta1) * gr;
      vf[k] = a.beta2 * vf[k] + (1.f - a.beta2) * gr * gr;
      const float denom = sqrtf(vf[k]) / a.biasCorr2Sqrt + a.eps;
      wf[k] = wf[k] * (1.f - a.lr * a.weightDecay) - (a.lr / a.biasCorr1) * (mf[k] / denom);
      p[k] = __float2bfloat16_rn(wf[k]);
    }
    st8<WIDE>(a.master + 8 * i, wf);
    st8<WIDE>(a.expAvg + 8 * i, mf);
    st8<WIDE>(a.expAvgSq + 8 * i, vf);
    reinterpret_cast<uint4*>(a.param)[i] = pq;
    if (a.zeroGrad) reinterpret_cast<uint4*>(const_cast<__nv_bfloat16*>(a.grad))[i] = make_uint4(0, 0, 0, 0);
  }
  // tail (n not a multiple of 8)
  for (uint64_t i = nVec * 8 + tid; i < a.n; i += nth) {
    const float gr = __bfloat162float(a.grad[i]) * a.gradScale;
    const float m = a.beta1 * a.expAvg[i] + (1.f - a.beta1) * gr;
    const float v = a.beta2 * a.expAvgSq[i] + (1.f - a.beta2) * gr * gr;
    const float denom = sqrtf(v) / a.biasCorr2Sqrt + a.eps;
    const float w = a.master[i] * (1.f - a.lr * a.weightDecay) - (a.lr / a.biasCorr1) * (m / denom);
    a.expAvg[i] = m; a.expAvgSq[i] = v; a.master[i] = w;
    a.param[i] = __float2bfloat16_rn(w);
    if (a.zeroGrad) const_cast<__nv_bfloat16*>(a.grad)[i] = __float2bfloat16_rn(0.f);
  }
}

}  // namespace

static mcclResult_t adamwLaunch(void* param, float* master, float* expAvg, float* expAvgSq, const void* grad,
                                uint64_t n, float lr, float beta1, float beta2, float eps, float weightDecay,
                                float gradScale, int step, int zeroGrad, const float* normSq, float maxNorm,
                                const float* hyper, mcclStream_t stream) {
  if (param == nullptr || master == nullptr || expAvg == nullptr || expAvgSq == nullptr || grad == nullptr || step < 1)
    return mcclInvalidArgument;
  if (n == 0) return mcclSuccess;
  // All five arrays are walked with 16/32-byte vectors.
  if (((uintptr_t)param | (uintptr_t)grad) & 15u || ((uintptr_t)master | (uintptr_t)expAvg | (uintptr_t)expAvgSq) & 15u)
    return mcclInvalidArgument;
  AdamArgs a;
  a.param = static_cast<__nv_bfloat16*>(param);
  a.master = master; a.expAvg = expAvg; a.expAvgSq = expAvgSq;
  a.grad = static_cast<const __nv_bfloat16*>(grad);
  a.n = n;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weightDecay = weightDecay; a.gradScale = gradScale;
  a.biasCorr1 = 1.f - powf(beta1, (float)step);
  a.biasCorr2Sqrt = sqrtf(1.f - powf(beta2, (float)step));
  a.zeroGrad = zeroGrad;
  a.normSq = normSq;
  a.maxNorm = maxNorm;
  a.hyper = hyper;
  const uint64_t vec = (n + 7) / 8;
  // One vector of eight elements per thread and no loop: with eight blocks per SM walking the array the last turn of the
  // walk leaves most of them idle (25 MB bucket: 63.7 us, 64 Mi elements: 314 us; without the walk 58.0 and 275 us).
  const uint64_t want = (vec + 255) / 256;
  const unsigned blocks = (unsigned)(want < (1u << 30) ? want : (1u << 30));
  const bool wide = (((uintptr_t)master | (uintptr_t)expAvg | (uintptr_t)expAvgSq) & 31u) == 0;
  auto* kernel = wide ? adamwKernel<true> : adamwKernel<false>;
  kernel<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
  return cudaGetLastError() == cudaSuccess ? mcclSuccess : mcclSystemError;
}

extern "C" mcclResult_t mcclFusedAdamW(void* param, float* master, float* expAvg, float* expAvgSq, const void* grad,
                                       uint64_t n, float lr, float beta1, float beta2, float eps, float weightDecay,
                                       float gradScale, int step, int zeroGrad, const float* normSq, float maxNorm,
                                       mcclStream_t stream) {
  return adamwLaunch(param, master, expAvg, expAvgSq, grad, n, lr, beta1, beta2, eps, weightDecay, gradScale, step, zeroGrad,
                     normSq, maxNorm, nullptr, stream);
}

// The same step with the learning rate and the two bias corrections read from device memory when the kernel
// runs: hyper = {lr, 1 - beta1^t, sqrt(1 - beta2^t)}.  For launches recorded in a CUDA graph.
extern "C" mcclResult_t mcclFusedAdamWDeviceHyper(void* param, float* master, float* expAvg, float* expAvgSq, const void* grad,
                                                  uint64_t n, const float* hyper, float beta1, float beta2, float eps,
                                                  float weightDecay, float gradScale, int zeroGrad, const float* normSq,
                                                  float maxNorm, mcclStream_t stream) {
  if (hyper == nullptr) return mcclInvalidArgument;
  return adamwLaunch(param, master, expAvg, expAvgSq, grad, n, 0.f, beta1, beta2, eps, weightDecay, gradScale, 1, zeroGrad,
                     normSq, maxNorm, hyper, stream);
}
