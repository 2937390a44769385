// fmf::make_snap and fmf::snapped against the two comparisons they stand for, in their
// order: prints the mismatches.
#include <cstdio>
#include <limits>
#include <random>

#include "snap.cuh"

int main() {
  std::mt19937_64 r(5);
  long bad = 0;
  auto check = [&](const fmf::Snap& s, double eps, double p) {
    double want = p;
    if (want <= eps) want = 0.0;
    if (1.0 - want <= eps) want = 1.0;
    long long b;
    std::memcpy(&b, &p, 8);
    const double got = fmf::snapped(p, b, s);
    bad += std::isnan(want) ? !std::isnan(got) : !(got == want);
  };
  const double inf = std::numeric_limits<double>::infinity();
  auto all = [&](double eps) {
    const fmf::Snap s = fmf::make_snap(eps);
    for (double at : {0.0, eps, 1.0 - eps, 0.5, 1.0})  // 40 doubles to either side
      for (double to : {-inf, inf}) {
        double p = at;
        for (int t = 0; t < 40; ++t, p = std::nextafter(p, to)) check(s, eps, p);
      }
    for (double p : {-0.0, -1.0, 2.0, -inf, inf, std::nan("")}) check(s, eps, p);
    for (int t = 0; t < 2000; ++t) {
      check(s, eps, (double)(r() >> 11) * 0x1p-53);
      long long b = (long long)r();
      double p;
      std::memcpy(&p, &b, 8);
      check(s, eps, p);
    }
  };
  // eps_trunc of solphi_mthinc1.f over sharp, flat and reversed profiles
  for (double bet : {300.0, 16.0, 8.0, 6.5, 4.0, 3.5, 2.0, 1.0, 0.5, 0.01, 0.0, -0.01, -0.5, -2.0, -3.0, -5.0, -7.0,
                     -7.5, -7.6, -7.7, -8.0, -300.0, inf, -inf, std::nan("")})
    all(0.5 * (std::tanh(-bet * 2.5) + 1.0));
  for (double eps : {5e-324, 1e-300, 1e-17, 0.5 - 0x1p-54, 0.5 + 0x1p-53, 1.0 - 0x1p-53, 1.5}) all(eps);
  std::printf("%ld\n", bad);
}
