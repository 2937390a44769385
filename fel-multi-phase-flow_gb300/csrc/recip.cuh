// recip.cuh -- reciprocal and reciprocal square root of a positive normal double
// without a division or a square root.
#pragma once

namespace fmf {

// The Newton-Raphson iteration for 1/x, r <- r + r (1 - x r), doubles the number
// of correct bits per step (P. Markstein, IBM J. Res. Develop. 34 (1990) 111-119);
// it starts here from the PTX approximate reciprocal rcp.approx.ftz.f64, and two
// steps reach double precision.  Inputs must be positive normal numbers (no
// subnormals, zero, infinity or NaN).  fmf_check_reciprocal measures its error
// and recip_h's against the IEEE quotient 1.0 / x.
__device__ __forceinline__ double recip_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

// 1/x by one third-order step, r <- r + r (e + e^2) with e = 1 - x r (the series
// 1/(1 - e) = 1 + e + e^2 + ..., E. Schroeder, Math. Ann. 2 (1870) 317-365): the
// approximate reciprocal, which reads the upper word of x alone, is within 2^-19.9
// (measured over 2^26 inputs, half of them with a low word of ones), its cube below 2^-59,
// so three FP64 operations give what recip_nr's four do.  Inputs and check as recip_nr.
__device__ __forceinline__ double recip_h(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// 1/sqrt(s) by one third-order step from the PTX approximate reciprocal square root
// rsqrt.approx.ftz.f64 (y, within 2^-20.0 as measured likewise): with e = 1 - s y^2 the
// binomial series gives 1/sqrt(s) = y (1 - e)^(-1/2) = y (1 + e/2 + 3/8 e^2 + 5/16 e^3 ...),
// |e| is below 2^-19 and the first term left out below 2^-58.  Five FP64 operations instead
// of a square root and a division.  Inputs as recip_nr.  fmf_check_rsqrt measures its error
// against 1.0 / sqrt(s).
__device__ __forceinline__ double rsqrt_h(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  const double e = fma(-(s * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

}  // namespace fmf
