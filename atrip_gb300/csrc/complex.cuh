// Complex FP64 arithmetic of the complex-field kernels.
#pragma once

#include <cuda_runtime.h>

namespace atrip_gb300 {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
  return c;
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cscale(double s, double2 a) {
  return make_double2(s * a.x, s * a.y);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
// Real part of a / d (Smith's algorithm).
__device__ __forceinline__ double cdiv_re(double2 a, double2 d) {
  if (fabs(d.y) <= fabs(d.x)) {
    const double r = d.y / d.x, den = d.x + d.y * r;
    return (a.x + a.y * r) / den;
  }
  const double r = d.x / d.y, den = d.x * r + d.y;
  return (a.x * r + a.y) / den;
}

}  // namespace
}  // namespace atrip_gb300
