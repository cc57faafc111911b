// Per-storage-form choices shared by the solver and the strip engine: the physics policy of the
// step kernels (exact for plain FP32 / FP64, fast for the 16-bit forms), its packed twin, the
// arithmetic of the moment pass, the per-launch constants, and the host equilibrium.
#pragma once

#include "collide.h"
#include "lbm_device.cuh"
#include "step_kernel.cuh"

namespace lbm_b200 {

template <class ST>
struct Form;
template <>
struct Form<float> {
  using A = ExactF32;
  using Phys = ExactPhys<ExactF32>;
  using PackedPhys = ExactPhysF32x2;
  static Phys::Consts consts(double tau, double fx, double fy) {
    return make_collide_consts<float>(float(tau), float(fx), float(fy));
  }
};
// FP64 with its multiplications on the integer units, for the kernels that the automatic choice
// takes (step kernels chosen by number keep the hardware's).
using F64IntPhys = ExactPhys<ExactF64Int>;
template <>
struct Form<double> {
  using A = ExactF64;
  using Phys = ExactPhys<ExactF64>;
  using PackedPhys = Phys;
  static Phys::Consts consts(double tau, double fx, double fy) {
    return make_collide_consts<double>(tau, fx, fy);
  }
};
template <>
struct Form<__half> {
  using A = ExactF32;  // moment pass
  using Phys = FastPhys;
  using PackedPhys = Phys;  // already packed
  static Phys::Consts consts(double tau, double fx, double fy) {
    return make_fast_consts(float(tau), float(fx), float(fy), kStoreScale16);
  }
};
template <>
struct Form<__nv_bfloat16> {
  using A = ExactF32;
  using Phys = FastPhys;
  using PackedPhys = Phys;  // already packed
  static Phys::Consts consts(double tau, double fx, double fy) {
    return make_fast_consts(float(tau), float(fx), float(fy), kStoreScale16);
  }
};

// Blocks per SM of the FP64 ring's grid. The collision is bound by the FP64 pipe, so what costs is
// an uneven last wave: more blocks than reside (two or three) let the scheduler hand out the
// last tiles one by one (1024 x 512 with the hardware's multiplications: 2702 MLUPS with the
// resident grid, 3065 with 6 per SM; with integer ones 4499 and, with 12 per SM, 4721).
constexpr int kF64GridPerSm = 12;

// Dynamic shared memory that keeps a kernel to `blocks` resident blocks per SM (228 KB per SM,
// 1 KB of it reserved per block).
inline size_t smem_for_blocks(int blocks) { return (228 * 1024 / static_cast<size_t>(blocks > 0 ? blocks : 1) - 1024) / 128 * 128; }

// Do 2048-cell tiles suit 16-bit rows of nx cells? They do unless a part-filled last tile costs more
// than the wider tiles gain over 1024-cell ones (MLUPS, 2048 / 1024: 3000 cells, 73 % / 98 % full,
// 136.6k / 165.1k; 5000, 81 % / 98 %, 165.6k / 166.0k; 3500, 85 % / 85 %, 151.6k / 141.5k).
inline bool wide_tiles16(int nx) {
  const long long wide = (nx + 2047LL) / 2048 * 2048, narrow = (nx + 1023LL) / 1024 * 1024;
  return nx >= 2048 && 20 * narrow >= 17 * wide;
}

inline constexpr int kCx[kQ] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
inline constexpr int kCy[kQ] = {0, 0, 1, 0, -1, 1, 1, -1, -1};

// Shifted equilibrium of (rho0, ux0, uy0) in T, the reference's expressions and order
// (src/common/boundary.hpp:26-34, src/common/d2q9.hpp:40-42).
template <class T>
inline Eq9<T> host_equilibrium(T rho0, T ux0, T uy0) {
  Eq9<T> e{};
  const T usq = ux0 * ux0 + uy0 * uy0;
  const T drho0 = rho0 - T(1);
  for (int i = 0; i < kQ; ++i) {
    const T cu = kCx[i] * ux0 + kCy[i] * uy0;
    e.v[i] = weight<T>(i) * (drho0 + rho0 * (T(3) * cu + T(4.5) * cu * cu - T(1.5) * usq));
  }
  return e;
}

}  // namespace lbm_b200
