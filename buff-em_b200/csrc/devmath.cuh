// Device arithmetic shared by the kernels.
#pragma once

// 1/sqrt(x) for normal positive x: the hardware approximation y (about 2^-22)
// and one step of Householder's iteration of order three (A. S. Householder, The
// Numerical Treatment of a Single Nonlinear Equation, 1970) for y^-2 - x,
//   y + y e (1/2 + 3/8 e),  e = 1 - x y^2,
// which is the binomial series of (1 - e)^{-1/2} cut after e^2 (omitted: 5/16 e^3,
// below 2^-64).  Five FP64 operations without a branch, so the point loops that
// call it can be interleaved.  Relative error at most 1.5 2^-53 (x y rounded once,
// 2^-53 in e, half of that in the result; the last operation 2^-53).
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = x * y, e = fma(-h, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// cos x and sin x for |x| <= 1: Taylor series at y = x/2 in Horner form (one
// fused multiply-add per term), then cos x = c^2 - s^2, sin x = 2 c s.  Terms
// to y^14 / y^15: the first omitted terms, y^16/16! and y^17/17!, are below
// 1e-18 for |y| <= 1/2.  cossin_small_short serves |x| <= 1/4 with the series
// of x itself, terms to x^12 / x^11 (first omitted terms x^14/14! and
// x^13/13!, below 5e-20 and 3e-18).
#define EXPI_C(n, f) (((n) & 1 ? -1.0 : 1.0) / (f))
__device__ __forceinline__ void cossin_small(double x, double &co, double &si) {
  const double y = 0.5 * x, y2 = y * y;
  double c = EXPI_C(7, 87178291200.0);           // 1/14!
  c = fma(c, y2, EXPI_C(6, 479001600.0));        // 1/12!
  c = fma(c, y2, EXPI_C(5, 3628800.0));
  c = fma(c, y2, EXPI_C(4, 40320.0));
  c = fma(c, y2, EXPI_C(3, 720.0));
  c = fma(c, y2, EXPI_C(2, 24.0));
  c = fma(c, y2, EXPI_C(1, 2.0));
  c = fma(c, y2, 1.0);
  double sn = EXPI_C(7, 1307674368000.0);        // 1/15!
  sn = fma(sn, y2, EXPI_C(6, 6227020800.0));     // 1/13!
  sn = fma(sn, y2, EXPI_C(5, 39916800.0));
  sn = fma(sn, y2, EXPI_C(4, 362880.0));
  sn = fma(sn, y2, EXPI_C(3, 5040.0));
  sn = fma(sn, y2, EXPI_C(2, 120.0));
  sn = fma(sn, y2, EXPI_C(1, 6.0));
  sn = fma(sn, y2, 1.0) * y;
  co = c * c - sn * sn;
  si = 2.0 * c * sn;
}
__device__ __forceinline__ void cossin_small_short(double x, double &co, double &si) {
  const double x2 = x * x;
  double c = EXPI_C(6, 479001600.0);             // 1/12!
  c = fma(c, x2, EXPI_C(5, 3628800.0));
  c = fma(c, x2, EXPI_C(4, 40320.0));
  c = fma(c, x2, EXPI_C(3, 720.0));
  c = fma(c, x2, EXPI_C(2, 24.0));
  c = fma(c, x2, EXPI_C(1, 2.0));
  co = fma(c, x2, 1.0);
  double sn = EXPI_C(5, 39916800.0);             // 1/11!
  sn = fma(sn, x2, EXPI_C(4, 362880.0));
  sn = fma(sn, x2, EXPI_C(3, 5040.0));
  sn = fma(sn, x2, EXPI_C(2, 120.0));
  sn = fma(sn, x2, EXPI_C(1, 6.0));
  si = fma(sn, x2, 1.0) * x;
}
