// Host check of the hand-over from integer to hardware multiplications (csrc/mul64.h, collide.h): a
// collision with integer products, done again where a result or the velocity is not finite, gives
// the hardware's numbers for every state, those of zero density and of infinite or NaN populations
// among them. Exit status 0 when all hold.
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>

#include "collide.h"
#include "mul64.h"

using namespace lbm_b200;

namespace {
struct IntArith : HostArith<double> {
  static double mul(double a, double b) { return mul64(a, b); }
};
constexpr double kInf = std::numeric_limits<double>::infinity();
constexpr double kNan = std::numeric_limits<double>::quiet_NaN();
long bad = 0;

bool same(double a, double b) { return std::isfinite(a) == std::isfinite(b) && (!std::isfinite(a) || a == b); }

void compare(const char* what, const double (&hw)[kQ], double (&in)[kQ], double ux) {
  bool again = !std::isfinite(ux);
  for (double v : in) again |= !std::isfinite(v);
  if (again) return;  // the kernels take the hardware's products for this cell
  for (int i = 0; i < kQ; ++i)
    if (!same(hw[i], in[i])) {
      std::printf("%s, direction %d: hardware %g, integer %g\n", what, i, hw[i], in[i]);
      ++bad;
      return;
    }
}

template <int K>
void collide(const double (&g)[kQ], double fx, double fy) {
  const CollideConsts<double> k = make_collide_consts<double>(0.7, fx, fy);
  double hw[kQ], in[kQ];
  collide_exact_kind<HostArith<double>, K>(g, k, hw);
  const double ux = collide_exact_kind<IntArith, K>(g, k, in);
  compare("collision", hw, in, ux);
  for (double alpha : {0.0, 0.1, -2.0, 1e-200, kInf, kNan}) {
    collide_exact_drag<HostArith<double>>(g, k, alpha, hw);
    const double uxd = collide_exact_drag<IntArith>(g, k, alpha, in);
    compare("drag collision", hw, in, uxd);
  }
}
}  // namespace

int main() {
  // States of zero density (one population -1, or -1 in parts), and every single population replaced.
  double states[3][kQ] = {{-1}, {-0.5, -0.125, 0, -0.125, 0, -0.0625, -0.0625, -0.0625, -0.0625}, {0, 1e-3, -2e-3, 0, 5e-4, 0, 1e-4, 0, -3e-4}};
  for (auto& s : states)
    for (int i = -1; i < kQ; ++i)
      for (double v : {kInf, -kInf, kNan, 0.0, -1.0, 1e200, 1e-200}) {
        double g[kQ];
        for (int j = 0; j < kQ; ++j) g[j] = j == i ? v : s[j];
        collide<kForceNone>(g, 0.0, 0.0);
        collide<kForceX>(g, 1e-5, 0.0);
        collide<kForceXY>(g, 1e-5, -3e-6);
      }
  std::printf("%ld mismatches\n", bad);
  return bad == 0 ? 0 : 1;
}
