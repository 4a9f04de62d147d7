// Conversions between FP32 and FP64 from the bits. GB300 converts at its FP64 rate, two lanes per
// clock and SM, which bounds every pass that mixes the two; integer instructions run at 64.
#pragma once

namespace rsg {

__device__ __forceinline__ double f2d(float x) {  // (double)x
  const unsigned b = __float_as_uint(x), e = (b >> 23) & 0xffu;
  if (e - 1u >= 254u) return (double)x;  // zero, subnormal, infinity, NaN
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ double rn24(double x) {  // (double)(float)x
  const unsigned hi = (unsigned)__double2hiint(x), e = (hi >> 20) & 0x7ffu;
  if (e - 897u >= 253u) return (double)(float)x;  // not a normal float
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return __longlong_as_double((long long)((b + 0x0fffffffull + ((b >> 29) & 1ull)) & ~0x1fffffffull));
}
__device__ __forceinline__ float d2f(double x) {  // (float)x
  const unsigned hi = (unsigned)__double2hiint(x), e = (hi >> 20) & 0x7ffu;
  if (e - 897u >= 253u) return (float)x;
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  const unsigned m = (unsigned)((b + 0x0fffffffull + ((b >> 29) & 1ull)) >> 29);  // exponent (bias 1023) and 23 bits
  return __uint_as_float((hi & 0x80000000u) | (m - (896u << 23)));
}

}  // namespace rsg
