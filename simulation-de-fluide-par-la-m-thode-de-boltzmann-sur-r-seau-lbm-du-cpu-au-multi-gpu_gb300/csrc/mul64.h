// Correctly rounded double multiplication in 32-bit integer arithmetic.
//
// sm_103a executes two FP64 operations per SM and cycle, against 64 integer multiply-adds and 128
// simple integer operations: a kernel of exact FP64 arithmetic leaves nine in ten issue slots
// idle while the FP64 pipe is full. Doing the multiplications on the integer units instead
// halves the pipe's load and runs beside it.
//
// The method is the schoolbook one of IEEE 754 arithmetic: the 53-bit significands are multiplied
// exactly (four 32 x 32 -> 64 products; the second factor is held 11 bits up, so that the high 64
// bits of the 117-bit product hold 52 or 53 significant ones), normalised by one bit, and rounded
// to nearest even from the bits below. A factor of zero gives zero (of positive sign: the exact
// forms treat -0 as +0), also with an infinite or NaN one, which IEEE 754 makes NaN; other factors
// outside [2^-400, 2^400), infinities and NaNs give NaN. The collision checks its results and its
// velocity and takes the hardware's multiplications where one of them is not finite
// (collide_cell; telling 0 * inf apart in every product costs 2 % on the ring and 14 % on the
// direct kernel, 300 x 300 3270 -> 2800 MLUPS).
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define MUL64_HD __host__ __device__ __forceinline__
#else
#define MUL64_HD inline
#endif

namespace lbm_b200 {

namespace mul64_detail {
// High word of ((hi:lo) << s), s = 0 or 1.
MUL64_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << 1) | (lo >> 31) : hi;
#endif
}
MUL64_HD void split(double v, uint32_t& hi, uint32_t& lo) {
#if defined(__CUDA_ARCH__)
  hi = static_cast<uint32_t>(__double2hiint(v));
  lo = static_cast<uint32_t>(__double2loint(v));
#else
  uint64_t b;
  std::memcpy(&b, &v, 8);
  hi = static_cast<uint32_t>(b >> 32);
  lo = static_cast<uint32_t>(b);
#endif
}
MUL64_HD double join(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
  const uint64_t b = (static_cast<uint64_t>(hi) << 32) | lo;
  double v;
  std::memcpy(&v, &b, 8);
  return v;
#endif
}
// |v| in [2^-400, 2^400): the product of two such factors is normal.
MUL64_HD bool in_window(uint32_t hi) { return (hi & 0x7fffffffu) - ((1023u - 400u) << 20) < (800u << 20); }
}  // namespace mul64_detail

MUL64_HD double mul64(double a, double b) {
  using namespace mul64_detail;
  uint32_t ahi, alo, bhi, blo;
  split(a, ahi, alo);
  split(b, bhi, blo);
  const uint32_t ah = (ahi & 0xfffffu) | 0x100000u;
  const uint32_t bh = (((bhi & 0xfffffu) | 0x100000u) << 11) | (blo >> 21), bl = blo << 11;
  const uint64_t p0 = static_cast<uint64_t>(alo) * bl;
  const uint64_t p1 = static_cast<uint64_t>(alo) * bh + (p0 >> 32);
  const uint64_t p2 = static_cast<uint64_t>(ah) * bl + static_cast<uint32_t>(p1);
  const uint64_t h = static_cast<uint64_t>(ah) * bh + (p1 >> 32) + (p2 >> 32);  // in [2^51, 2^53)
  const uint32_t hh = static_cast<uint32_t>(h >> 32), hl = static_cast<uint32_t>(h);
  const uint32_t lh = static_cast<uint32_t>(p2), ll = static_cast<uint32_t>(p0);
  const uint32_t s = ((hh >> 20) & 1u) ^ 1u;
  const uint32_t mh = shl_hi(hl, hh, s), ml = shl_hi(lh, hl, s);
  const uint32_t rh = shl_hi(ll, lh, s), rl = ll << s;
  // Up when the rest is above one half, or is one half and the significand is odd.
  const uint32_t odd_or_rest = rl != 0u ? 1u : (ml & 1u);
  const uint64_t m = ((static_cast<uint64_t>(mh) << 32) | ml) + (rh > 0x80000000u - odd_or_rest ? 1u : 0u);
  // mh carries the implicit bit, which adds one to the exponent field.
  const uint32_t e = (ahi & 0xfff00000u) + (bhi & 0xfff00000u) - (s << 20) - (1023u << 20);
  const bool ok = in_window(ahi) && in_window(bhi);
  const bool zero = ((ahi & 0x7fffffffu) | alo) == 0u || ((bhi & 0x7fffffffu) | blo) == 0u;
  const uint32_t hi = ok ? static_cast<uint32_t>(m >> 32) + e : (zero ? 0u : 0x7ff80000u);
  return join(hi, ok ? static_cast<uint32_t>(m) : 0u);
}

}  // namespace lbm_b200
