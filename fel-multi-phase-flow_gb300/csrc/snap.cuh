// snap.cuh -- the snap of phi to 0 or 1 outside the interface band (solphi_mthinc1.f,
// solphi_mthinc3.f) as tests on its bits: a double comparison takes a slot of the FP64 pipe.
#pragma once
#include <cmath>
#include <cstring>

#if defined(__CUDACC__)
#define SNAP_FN __host__ __device__ __forceinline__
#else
#define SNAP_FN inline
#endif

namespace fmf {

// The two statements "p <= eps: p = 0", "1 - p <= eps: p = 1" in that order: p with bits at
// or below `low` becomes `below`, else with bits at or above `high` 1.  (eps = (1 -
// tanh(2.5 beta))/2 is below 1/2 for beta > 0; it reaches 1 at beta = -7.6, where the second
// statement takes up what the first one leaves.)
struct Snap {
  long long low, high;
  double below;
};
inline Snap make_snap(double eps) {
  Snap s{};
  if (std::isnan(eps)) return {(long long)0x8000000000000000ull, 0x7fffffffffffffffll, 0.0};  // no comparison holds
  std::memcpy(&s.low, &eps, sizeof eps);
  if (eps >= 1.0) {
    s.below = 1.0;
    return s;
  }
  // the smallest t with 1 - t <= eps, by bisection over the bits of (0, 1]: 1 - t never
  // grows with t, and neighbouring doubles have neighbouring bits
  long long lo = 0, hi = 0x3ff0000000000000ll;
  while (hi - lo > 1) {
    const long long mid = lo + (hi - lo) / 2;
    double t;
    std::memcpy(&t, &mid, sizeof t);
    (1.0 - t <= eps ? hi : lo) = mid;
  }
  s.high = hi;
  return s;
}
// p, whose bits are b; NaN stays
SNAP_FN double snapped(double p, long long b, const Snap& s) {
  if (((unsigned long long)b << 1) > 0xffe0000000000000ull) return p;
  if (b <= s.low) return s.below;
  return b >= s.high ? 1.0 : p;
}

}  // namespace fmf
