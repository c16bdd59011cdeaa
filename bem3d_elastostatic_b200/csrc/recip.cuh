// 1/sqrt(x), 1/x and v/p from the hardware's approximations of their leading bits, in fewer
// operations than CUDA's own functions take: they sit in loops that the FP64 pipe or one chain of
// latencies bounds.  The bounds below are relative errors, u = 2^-53 (FP64) or 2^-24 (FP32).
#pragma once

namespace bem {

// 1 / sqrt(x), by the binomial series: with y the approximation and e = 1 - x y^2,
// 1 / sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3/8 e^2) + 5/16 e^3 y ...  For |e| < 2^-18
// (measured 2^-19.1) the rest is 0.16 u, the rounding of x y adds u/2 and the last operation u:
// below 1.7 u (measured 1.24 u; CUDA's rsqrt is within 1 ulp, up to 2 u).  Normal x.  Five FP64
// operations.
__device__ __forceinline__ double rsqrt_h3(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ float rsqrt_h3(float x) { return rsqrtf(x); }

// 1 / x by the geometric series (the hyperpower iteration of order three, Altman 1960): with e =
// 1 - x y, 1 / x = y / (1 - e) = y (1 + e + e^2) + e^3 y ...  For |e| < 2^-18 (measured 2^-20.0)
// the rest is u/2: below 1.6 u (measured 1.00 u).  Normal x and 1/x.
__device__ __forceinline__ double reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float reciprocal(float x) { return __frcp_rn(x); }

// 1 / x in FP32 by one Newton step from the approximation (within 1 ulp, so that the step's e^2
// is far below rounding): below 1.01 u (measured 1.00 u).  Normal x, 1/x.
__device__ __forceinline__ float reciprocal_newton(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return fmaf(y, fmaf(-x, y, 1.f), y);
}

// v / p from r, 1 / p to a few u: the product with r, corrected once by its remainder (Markstein
// 1990, IBM J. Res. Dev. 34): the remainder is exact, so the last operation's rounding is all of
// the error: u (1 + 2^-10) for v, p and v / p far from the ends of the exponent range (measured: the
// correctly rounded quotient in each of 2^21 cases of either type).
template <typename T>
__device__ __forceinline__ T corrected_quotient(T v, T p, T r) {
  const T l = v * r;
  return fma(fma(-l, p, v), r, l);
}

}  // namespace bem
