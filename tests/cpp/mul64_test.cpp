// Host check of the integer double multiplication (csrc/mul64.h) against the processor's: random
// factors over the window of exponents, factors with few and with nearly all significant bits
// (ties and carries), the collision's constants, zeros, the window's edges, and NaN outside it.
// Exit status 0 when every product is equal.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

#include "mul64.h"

int main() {
  std::mt19937_64 r(1);
  long bad = 0;
  auto check = [&](double a, double b) {
    const double want = a * b, got = lbm_b200::mul64(a, b);
    if (!(want == got)) {
      if (bad < 10) std::printf("%a * %a = %a, got %a\n", a, b, want, got);
      ++bad;
    }
  };
  for (long k = 0; k < 4000000; ++k) {
    const int mode = static_cast<int>(k % 6);
    auto make = [&] {
      uint64_t v = r();
      if (mode == 1) v &= ~((1ull << 26) - 1);
      if (mode == 2) v &= ~((1ull << (v >> 58)) - 1);
      if (mode == 3) v |= (1ull << 30) - 1;
      const int e = mode == 4 ? static_cast<int>(r() % 800) - 400 : static_cast<int>(r() % 120) - 60;
      const uint64_t b = (v & 0x800fffffffffffffull) | (static_cast<uint64_t>(1023 + e) << 52);
      double d;
      std::memcpy(&d, &b, 8);
      return d;
    };
    const double a = make(), b = make();
    check(a, b);
    if (mode == 5)
      for (double c : {3.0, 9.0, 1.5, 1.0 / 9, 4.0 / 9, 1.0 / 36}) check(a, c);
  }
  for (double z : {0.0, -0.0})
    for (double b : {1.0, -3.5, 1e-300, 1e300, 0.0}) check(z, b), check(b, z);
  const double lo = std::ldexp(1.0, -400), hi = std::ldexp(1.0, 400), one = 1.0 + std::ldexp(1.0, -52),
               two = 2.0 - std::ldexp(1.0, -52);
  for (double a : {lo, std::nextafter(hi, 0.0), 1.0, one, two})
    for (double b : {lo, std::nextafter(hi, 0.0), 1.0, -one, two}) check(a, b);
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  for (double a : {std::nextafter(lo, 0.0), hi, inf, -inf, nan, std::numeric_limits<double>::denorm_min()})
    if (!std::isnan(lbm_b200::mul64(a, 1.5)) || !std::isnan(lbm_b200::mul64(1.5, a))) ++bad;
  std::printf("%ld mismatches\n", bad);
  return bad == 0 ? 0 : 1;
}
