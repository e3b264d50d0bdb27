// Device arithmetic shared by the kernels.
#pragma once

// 1/sqrt(x) for normal positive x: the hardware approximation (about 2^-22)
// and one step of the third-order iteration y + y e (1/2 + 3/8 e),
// e = 1 - x y^2 (the binomial series of (1 - e)^{-1/2}; what it omits is
// 5/16 e^3, below 2^-64).  Five FP64 operations without a branch, so the point
// loops that call it can be interleaved; within 2 ulp of the exact value.
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = x * y, e = fma(-h, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
