// Double-double arithmetic (pairs hi + lo, |lo| <= ulp(hi)/2), used where tables are
// built so that the stored doubles are correctly rounded (device code).
#pragma once

#include <cuda_runtime.h>

namespace s2g {
namespace {

struct dd {
  double hi, lo;
};
__device__ __forceinline__ dd dd_quick(double a, double b) {
  const double s = a + b;
  return dd{s, b - (s - a)};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
  const double s = a.hi + b.hi, bb = s - a.hi;
  const double e = (a.hi - (s - bb)) + (b.hi - bb) + a.lo + b.lo;
  return dd_quick(s, e);
}
__device__ __forceinline__ dd dd_neg(dd a) { return dd{-a.hi, -a.lo}; }
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
  const double p = a.hi * b.hi;
  double e = fma(a.hi, b.hi, -p);
  e = fma(a.hi, b.lo, e);
  e = fma(a.lo, b.hi, e);
  return dd_quick(p, e);
}
__device__ __forceinline__ dd dd_mul_d(dd a, double b) {
  const double p = a.hi * b;
  double e = fma(a.hi, b, -p);
  e = fma(a.lo, b, e);
  return dd_quick(p, e);
}
__device__ __forceinline__ dd dd_div(dd a, dd b) {
  const double q1 = a.hi / b.hi;
  dd r = dd_add(a, dd_neg(dd_mul_d(b, q1)));
  const double q2 = r.hi / b.hi;
  r = dd_add(r, dd_neg(dd_mul_d(b, q2)));
  const double q3 = r.hi / b.hi;
  return dd_add(dd_quick(q1, q2), dd{q3, 0.0});
}
// sqrt of an exactly representable double, to double-double accuracy
__device__ __forceinline__ dd dd_sqrt_d(double x) {
  const double r = sqrt(x);
  if (r == 0.0) return dd{0.0, 0.0};
  return dd_quick(r, fma(-r, r, x) / (2.0 * r));
}

}  // namespace
}  // namespace s2g
