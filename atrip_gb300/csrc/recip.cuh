// The split forms' FP64 helpers: exact conversions and the reciprocal of an
// energy denominator.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace atrip_gb300 {
namespace {

__device__ __noinline__ double recip_div(double d) { return 1.0 / d; }

// Exact conversions to FP64 done with integer instructions.  The energy
// warps are bound by this GPU's narrow FP64 pipe; integer operations run
// beside it.
// |n| < 2^51: 1.5 2^52 + n has ulp 1, so its bit pattern is that of
// 1.5 2^52 plus n in the low mantissa bits; subtracting 1.5 2^52 is exact.
__device__ __forceinline__ double i64_to_f64_exact(long long n) {
  return __longlong_as_double(0x4338000000000000ll + n) - 6755399441055744.0;
}
// Normal FP32 values: same sign and mantissa, exponent rebiased (127 ->
// 1023); zero, subnormal, infinity and NaN take the conversion instruction.
__device__ __forceinline__ double f32_to_f64_exact(float f) {
  const uint32_t u = __float_as_uint(f);
  const uint32_t e = (u >> 23) & 0xffu;
  if (e == 0u || e == 0xffu) return (double)f;
  const unsigned long long bits = ((unsigned long long)(u & 0x80000000u) << 32) |
                                  ((unsigned long long)(e + 896u) << 52) |
                                  ((unsigned long long)(u & 0x7fffffu) << 29);
  return __longlong_as_double((long long)bits);
}

// 1/d for the energy denominators: d truncated to FP32 (integer
// operations), its FP32 reciprocal (rounded to nearest), widened exactly,
// refined by one Newton-Raphson step x1 = x0 + x0 (1 - d x0) in FP64.
// With |x0 d - 1| <= ~1.5 2^-23 the relative error of x1 is about its
// square (< 2^-44) plus one rounding; outside the FP32 exponent range it
// falls back to the division (out of line: the orbital-energy gaps never
// get there).
__device__ __forceinline__ double recip_nr(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const int e = (int)((b >> 52) & 0x7ffu) - 1023;
  if (e < -125 || e > 126) return recip_div(d);
  const uint32_t fb = ((uint32_t)(b >> 32) & 0x80000000u) | ((uint32_t)(e + 127) << 23) |
                      ((uint32_t)(b >> 29) & 0x7fffffu);
  const double x0 = f32_to_f64_exact(__frcp_rn(__uint_as_float(fb)));
  const double err = fma(-d, x0, 1.0);
  return fma(x0, err, x0);
}

}  // namespace
}  // namespace atrip_gb300
