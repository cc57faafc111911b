// Host check of the exact collision's short forms (csrc/collide.h) against the literal collision of
// the reference's v0 (src/v0_cpu/solver_v0.cpp:86-99,127-143, src/common/d2q9.hpp:40-50) where
// products underflow: populations and forces from the smallest subnormal number up, from rest and
// not, by the force kind that the library takes for them, in float and double, over a few steps of
// one cell's own populations.
// Exit status 0 when every output value is equal. Compile with -ffp-contract=off.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "collide.h"

namespace {

constexpr int CX[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
constexpr int CY[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};

template <class T>
void literal(const T* g, T omega, T fp, T fx, T fy, T* out) {
  T m0 = 0, mx = 0, my = 0;
  for (int i = 0; i < 9; ++i) {
    m0 += g[i];
    mx += CX[i] * g[i];
    my += CY[i] * g[i];
  }
  const T drho = m0, rho = T(1) + drho;
  const T ux = (mx + T(0.5) * fx) / rho, uy = (my + T(0.5) * fy) / rho;
  const T usq = ux * ux + uy * uy;
  for (int i = 0; i < 9; ++i) {
    const T wi = lbm_b200::weight<T>(i), cxi = T(CX[i]), cyi = T(CY[i]);
    const T cu = cxi * ux + cyi * uy, cf = cxi * fx + cyi * fy;
    const T geq = wi * (drho + rho * (T(3) * cu + T(4.5) * cu * cu - T(1.5) * usq));
    const T guo = wi * (T(3) * ((cxi - ux) * fx + (cyi - uy) * fy) + T(9) * cu * cf);
    out[i] = g[i] - omega * (g[i] - geq) + fp * guo;
  }
}

// forces: components that may be non-zero (the force kinds' numbering).
template <class T>
long check(int forces, long trials, unsigned seed) {
  std::mt19937_64 rng(seed);
  const double lo = std::log2(double(std::numeric_limits<T>::denorm_min())), hi = -3.0;
  std::uniform_real_distribution<double> u(-1.0, 1.0), l(lo, hi);
  auto tiny = [&] { return T(std::copysign(std::exp2(l(rng)), u(rng))); };
  long bad = 0;
  for (long t = 0; t < trials; ++t) {
    const T fx = forces == lbm_b200::kForceNone ? T(0) : tiny();
    const T fy = forces == lbm_b200::kForceXY ? tiny() : T(0);
    const double common = l(rng);
    T g[9];
    for (int i = 0; i < 9; ++i) {
      const int mode = static_cast<int>(rng() % 8);
      g[i] = t % 3 == 0 || mode == 0 ? T(0) : (mode < 4 ? T(std::exp2(common) * u(rng)) : tiny());
    }
    // Momentum that nearly cancels the force's half, and little else.
    if (t % 5 == 0) {
      for (T& v : g) v = T(0);
      g[1] = T(-0.25) * fx;
      g[3] = T(0.25) * fx;
      g[1] = T(g[1] * (T(1) + T(rng() % 3) * std::numeric_limits<T>::epsilon()));
    }
    const auto k = lbm_b200::make_collide_consts<T>(T(0.501 + 0.7 * (1.0 + u(rng))), fx, fy);
    for (int step = 0; step < 4; ++step) {
      T a[9], b[9];
      literal<T>(g, k.omega, k.force_prefactor, fx, fy, a);
      lbm_b200::collide_exact<lbm_b200::HostArith<T>>(g, k, b);
      for (int i = 0; i < 9; ++i)
        if (!(a[i] == b[i])) {
          if (bad < 4)
            std::printf("kind %d, state %ld, step %d, direction %d: %.9g, literal %.9g (fx %.9g)\n", k.force, t, step, i,
                        double(b[i]), double(a[i]), double(fx));
          ++bad;
        }
      for (int i = 0; i < 9; ++i) g[i] = a[i];
    }
  }
  return bad;
}

template <class T>
long all() {
  const long n = 400000;
  return check<T>(lbm_b200::kForceNone, n, 1) + check<T>(lbm_b200::kForceX, n, 2) + check<T>(lbm_b200::kForceXY, n, 3);
}

}  // namespace

int main() {
  const long f = all<float>(), d = all<double>();
  std::printf("float %ld, double %ld mismatching values\n", f, d);
  return f == 0 && d == 0 ? 0 : 1;
}
