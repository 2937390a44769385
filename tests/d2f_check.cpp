// df::d2f against the conversion it stands in for: random bits, exponents around float's
// range, ties and their neighbours at every length of cut; prints the mismatches.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "df64.cuh"

int main() {
  std::mt19937_64 r(7);
  long bad = 0;
  auto check = [&](double x) {
    const float a = fmf::df::d2f(x), b = (float)x;
    bad += std::isnan(x) ? !std::isnan(a) : std::memcmp(&a, &b, 4) != 0;
  };
  auto of = [&](unsigned long long b) {
    double x;
    std::memcpy(&x, &b, 8);
    check(x);
  };
  for (long i = 0; i < 2000000; ++i) {
    unsigned long long b = r();
    of(b);
    b = (b & 0x800fffffffffffffull) | (860ull + r() % 310) << 52;
    of(b);
    const int cut = 29 + (int)(r() % 24);
    b &= ~((1ull << cut) - 1);
    of(b | 1ull << (cut - 1));
    of((b | 1ull << (cut - 1)) + 1);
    of((b | 1ull << (cut - 1)) - 1);
    of(b);
  }
  const double inf = INFINITY;
  for (double x : {0.0, 1e-45, 7e-46, 1.4e-45, 1.1754943508222875e-38, 3.4028235677973366e38, 1e39, inf, (double)NAN}) {
    check(x);
    check(-x);
  }
  std::printf("%ld\n", bad);
}
