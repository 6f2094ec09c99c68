// Cutting FP64 values into eight signed 8-bit digits (triples_fp64_tc.cu).
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace atrip_gb300 {
namespace {

// round(x 2^(63-e)) for |x| <= 127/128 2^e, with integer instructions.
__device__ __forceinline__ long long fixed63(double x, int e) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex == 0) return 0;  // zero or subnormal: below 2^(e-64) for any e accepted
  const long long m = (long long)((b & 0xfffffffffffffull) | 0x10000000000000ull);
  const int sh = ex - 1075 + 63 - e;  // <= 10
  long long v;
  if (sh >= 0) v = m << sh;
  else if (sh < -54) v = 0;
  else v = (m + (1ll << (-sh - 1))) >> -sh;
  return (long long)b < 0 ? -v : v;
}
// The bytes of X plus 128 in each of the seven lower ones: digit + 128.
__device__ __forceinline__ unsigned long long biased(long long X) {
  return (unsigned long long)X + 0x0080808080808080ull;
}
// Digit s of a biased value.
__device__ __forceinline__ float digit(unsigned long long y, int s) {
  if (s == 0) return (float)(int)((long long)y >> 56);
  return __uint_as_float(0x4B000000u | (uint32_t)((y >> (56 - 8 * s)) & 0xff)) - 8388736.f;
}

}  // namespace
}  // namespace atrip_gb300
