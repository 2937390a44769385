// bits.cuh -- tests on a double's bits.  A double comparison, minimum or maximum takes a
// slot of the FP64 pipe (64 cycles per warp and quarter SM on GB300); these do not.
#pragma once

namespace fmf {

constexpr long long kOneBits = 0x3ff0000000000000ll;  // 1.0
constexpr long long kInfBits = 0x7ff0000000000000ll;

// the magnitude bits shifted up: 0 for +0 and -0 only
__device__ __forceinline__ unsigned long long mag(double x) {
  return (unsigned long long)__double_as_longlong(x) << 1;
}
__device__ __forceinline__ bool is_nan(double x) { return mag(x) > ((unsigned long long)kInfBits << 1); }
__device__ __forceinline__ bool finite_bits(long long b) { return ((b >> 52) & 0x7ff) != 0x7ff; }
// x >= 0 (true for -0; differs from the comparison for NaN only)
__device__ __forceinline__ bool nonneg(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 || (b << 1) == 0;
}
// fmax(fmin(p, 1), 0): NaN gives 1, as fmin does; -0 gives 0
__device__ __forceinline__ double clip01(double p) {
  const long long b = __double_as_longlong(p);
  if (b > kOneBits || is_nan(p)) return 1.0;
  return b < 0 ? 0.0 : p;
}
// p <= eps gives 0 and 1 - p <= eps gives 1 (solphi_mthinc1.f, solphi_mthinc3.f): eps > 0 as
// bits, and the smallest double t with 1 - t <= eps as bits (one_minus, below)
__device__ __forceinline__ double snap01(double p, long long eps, long long one_eps) {
  const long long b = __double_as_longlong(p);
  if (is_nan(p)) return p;
  if (b <= eps) return 0.0;
  return b >= one_eps ? 1.0 : p;
}

}  // namespace fmf
