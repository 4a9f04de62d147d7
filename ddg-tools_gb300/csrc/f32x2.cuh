// Packed FP32 pairs.
#pragma once

namespace rsg {

// Two FP32 values in one 64-bit register (first in the low half) and the packed FP32 pair
// arithmetic of sm_100 and later (each half rounded to nearest, as the scalar operations).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
constexpr f32x2 kF2Sign = 0x8000000080000000ull;  // both halves' sign bits
__device__ __forceinline__ f32x2 f2_neg(f32x2 a) { return a ^ kF2Sign; }
// The same on one value, for code written for either. Sums rounded to nearest are never contracted with the
// product before them, so the product needs no such form (with __fmul_rn the energy's value takes 4 % longer).
__device__ __forceinline__ float f2_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float f2_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float f2_mul(float a, float b) { return a * b; }
__device__ __forceinline__ float f2_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float f2_neg(float a) { return -a; }
__device__ __forceinline__ f32x2 f2_dup(float a) { return f2_pack(a, a); }

}  // namespace rsg
