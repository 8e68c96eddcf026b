// Two fp32 operations per instruction (add, mul and fma .f32x2 of sm_100): the same roundings as one by one, half the issue slots.
// For the kernels that arithmetic bounds beside their memory traffic.
#pragma once

#include <stdint.h>

namespace mccl {

struct F2 { uint64_t v; };

__device__ __forceinline__ F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void split(F2 p, float* a, float* b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(p.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// Two bf16 numbers of a 32-bit word.
__device__ __forceinline__ F2 f2OfBf16(uint32_t w) { return f2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

}  // namespace mccl
