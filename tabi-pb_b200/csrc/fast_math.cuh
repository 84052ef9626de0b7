// fast_math.cuh -- the two functions of the FP64 pair kernels, which the FP64
// pipe bounds, in fewer of its instructions.
//
// e^-u for u >= 0 by a table and a short polynomial (Tang, "Table-driven
// implementation of the exponential function", ACM TOMS 15 (1989), with a
// table in u itself: kappa times a distance is small, so no reduction by ln 2
// is needed).
// u = k/32 + d, |d| <= 1/64: e^-u = T[k] + T[k] (e^-d - 1), e^-d - 1 by its Taylor
// polynomial of degree 6 (truncation 4.5e-17).  10 FP64 instructions and one
// shared load, against about 18 FP64 and 10 integer ones of exp(); within 1.5
// ulp of it where tested.  u >= 15.98, infinities and NaN take exp(); a caller
// that knows its u to be below kExpTabEnd leaves that test out (CHECK false).
//
// 1/sqrt(x) from the hardware's approximation y (relative error about 2^-20)
// and one third-order Householder step, y + y e (1/2 + 3/8 e) with e = 1 - x y^2
// (remaining error of the step 5/16 e^3 < 2^-59): 5 FP64 instructions, no branch.
// x = 0 gives NaN, not infinity; x below the smallest normal counts as 0.
#pragma once

namespace tabi {

constexpr int kExpTab = 512;  // entries: e^{-k/32}, u < 16
constexpr double kExpTabEnd = 15.98;

// fills the block's table; the caller synchronises
__device__ __forceinline__ void exp_table_fill(double* tab) {
  for (int k = threadIdx.x; k < kExpTab; k += blockDim.x) tab[k] = exp(-k * (1.0 / 32.0));
}

template <bool CHECK = true>
__device__ __forceinline__ double exp_neg(double u, const double* tab) {
  constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer
  // 0x402ff5c2 is the high word of 15.98; NaN and infinity are above it
  if (CHECK && __double2hiint(u) >= 0x402ff5c2) return exp(-u);
  const double t = fma(u, 32.0, kShift);
  const double d = fma(t - kShift, -1.0 / 32.0, u);
  const double T = tab[__double2loint(t) & (kExpTab - 1)];  // in bounds for a NaN too
  double p = fma(d, 1.0 / 720.0, -1.0 / 120.0);
  p = fma(p, d, 1.0 / 24.0);
  p = fma(p, d, -1.0 / 6.0);
  p = fma(p, d, 0.5);
  p = fma(p, d, -1.0);
  return fma(T, p * d, T);
}

__device__ __forceinline__ double fast_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

}  // namespace tabi
