// sgnb_fastmath.cuh -- the fast arithmetic mode's reciprocal and square root.
//
// Both refine a hardware estimate by the steps named below; the exact mode never uses them.
// Tested against the device's IEEE results in ulps (tests/test_fast_math_gpu.py,
// tests/test_fast_accuracy_gpu.py, through sgnb_fast_math).
#pragma once

namespace sgnb {
namespace dev {

// Reciprocal for the fast mode: the hardware estimate (PTX rcp.approx.ftz.f64, about 20 bits) refined
// by two Newton-Raphson steps r <- r + r (1 - x r), each of which doubles the number of correct
// bits. For normal x (the positive depths and error scales it is used on). One step of third
// order would save an operation, but reached 0.506 ulp where this stays at 0.5.
__device__ __forceinline__ double fast_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}

// Square root for the fast mode from the hardware estimate y of 1/sqrt(x) (PTX
// rsqrt.approx.ftz.f64): one step of third order, with e = 1 - x y^2 and s = x y,
// sqrt(x) = s (1 - e)^(-1/2) = s + s e (1/2 + 3/8 e) + O(e^3), then one Newton (Heron) step on
// s^2 = x written with the residual, s <- s + (y/2) (x - s^2), which takes the rounding of x y
// out again (0.76 -> 0.5 ulp). Normal finite x only.
__device__ __forceinline__ double fast_sqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double s = x * y;
  const double e = fma(-s, y, 1.0);
  s = fma(s * e, fma(0.375, e, 0.5), s);
  return fma(0.5 * y, fma(-s, s, x), s);
}
// The same for any x: zero, subnormal, infinite, negative and NaN arguments take the IEEE square
// root. Tested against IEEE sqrt in ulps through sgnb_fast_math.
__device__ __forceinline__ double fast_sqrt(double x) {
  if (!(x >= 2.2250738585072014e-308 && x <= 1.7976931348623157e308)) return sqrt(x);
  return fast_sqrt_normal(x);
}

}  // namespace dev
}  // namespace sgnb
