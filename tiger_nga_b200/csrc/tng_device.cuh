// Device helpers shared by the generated mechanism code and the kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

// Literal-mode select: LM == 0 keeps the reference build's literal kinds (default-real
// literals rounded to float32), LM == 1 reads every literal as a double.
#define TNG_LM(ref, dbl) (LM ? (dbl) : (ref))

namespace tng {

// 2^x on the FP32 special-function unit (ex2.approx, flushes subnormal results to zero).
__device__ __forceinline__ float tng_ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// log2(x) on the FP32 special-function unit; log2(0) = -inf.
__device__ __forceinline__ float tng_lg2f(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// log2(1 + 2^x) without overflow for large x.
__device__ __forceinline__ float tng_softplus2f(float x) {
  return fmaxf(x, 0.0f) + tng_lg2f(1.0f + tng_ex2f(-fabsf(x)));
}

// Packed FP32 pairs (sm_100 f32x2 instructions: one FMA / MUL / ADD for two values; each lane is
// rounded as the scalar instruction would round it). Element 0 in the low 32 bits.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float x, float y) {
  return (f32x2)__float_as_uint(x) | ((f32x2)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float f2_lo(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f2_hi(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

}  // namespace tng
