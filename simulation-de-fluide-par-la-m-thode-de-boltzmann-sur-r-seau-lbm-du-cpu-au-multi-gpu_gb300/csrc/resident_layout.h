// How a grid is cut into tiles for the resident step kernel (step_resident.cuh), and where a
// tile's edge values go. Plain C++ so that the host checks the exchange (tests) with the code
// the kernel runs.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#if defined(__CUDACC__)
#define RES_HD __host__ __device__ __forceinline__
#else
#define RES_HD inline
#endif

namespace lbm_b200 {

constexpr int kResPlaneBytes = 11648;          // of one plane of one buffer (2 x 9 of them)
constexpr int kResMaxItems = 512, kResMaxMask = 1024, kResMaxWords = 800;
constexpr size_t kResSmemBytes =
    18 * static_cast<size_t>(kResPlaneBytes) + 12 * kResMaxWords + 4 * kResMaxMask + 4 * kResMaxItems;
static_assert(kResSmemBytes <= 227 * 1024, "shared memory of one block");

// How a grid is cut: tx x ty tiles; every tile is `w` cells wide except the last of a row, and
// rows are split evenly (the first `extra` bands one row more).
struct ResLayout {
  int tx = 0, ty = 0, w = 0, base = 0, extra = 0;
  int hs = 0, ws = 0;  // outbox strides: rows and row words of the largest tile
  RES_HD int words() const { return 2 * (hs + ws); }  // outbox words per tile and parity
  RES_HD int width(int cx, int nx) const { return cx == tx - 1 ? nx - cx * w : w; }
  RES_HD int height(int cy) const { return base + (cy < extra ? 1 : 0); }
  RES_HD int row0(int cy) const { return cy * base + (cy < extra ? cy : extra); }
};

// Element stride of a buffer row and the column of cell 0 in it. 16-bit rows keep cell pairs on
// 4-byte boundaries.
template <int kElem>
RES_HD constexpr int res_stride(int w) {
  return kElem == 2 ? ((w + 1) & ~1) + 4 : w + 2;
}
template <int kElem>
RES_HD constexpr int res_col0() {
  return kElem == 2 ? 2 : 1;
}
// Outbox words of a row of w cells, and words polled per step for a w x h tile.
template <int kElem>
RES_HD constexpr int res_row_words(int w) {
  return kElem == 2 ? (w + 1) / 2 : w;
}
template <int kElem>
RES_HD constexpr int res_polls(int w, int h) {
  return 2 * (res_row_words<kElem>(w) + h) + 4;
}

// Outbox of a tile, in words of three values (the planes that cross that edge) and the tag:
// E [hs] planes 1, 5, 8 of the last column, W [hs] 3, 6, 7 of the first, N [ws] 2, 5, 6 of the top
// row, S [ws] 4, 7, 8 of the bottom row.
RES_HD int res_off_e(const ResLayout&) { return 0; }
RES_HD int res_off_w(const ResLayout& L) { return L.hs; }
RES_HD int res_off_n(const ResLayout& L) { return 2 * L.hs; }
RES_HD int res_off_s(const ResLayout& L) { return 2 * L.hs + L.ws; }

// One entry of a tile's poll list: the word (offset over all tiles, one parity), the element
// offsets its three values go to (kPollSkip: not needed) and how they are stored.
constexpr uint16_t kPollSkip = 0xffff;
constexpr uint16_t kPollWord = 0, kPollLow = 1, kPollHigh = 2;
struct PollEntry {
  uint32_t src;
  uint16_t d[3], kind;
};
static_assert(sizeof(PollEntry) == 12 && 9 * kResPlaneBytes / 2 < kPollSkip, "poll entries");

// e = 0 .. res_polls - 1: row -1 from the tile below (its N), row h from the tile above (its S),
// column -1 from the left (its E), column w from the right (its W), then the corners: plane 5
// from below left, 6 from below right, 8 from above left, 7 from above right.
template <int kElem>
RES_HD PollEntry res_poll_entry(const ResLayout& L, int nx, int cx, int cy, int w, int h, int e) {
  constexpr int PS = kResPlaneBytes / kElem;
  constexpr bool k16 = kElem == 2;
  const int rs = res_stride<kElem>(w), c0 = res_col0<kElem>(), rw = res_row_words<kElem>(w);
  const int xw = cx == 0 ? L.tx - 1 : cx - 1, xe = cx == L.tx - 1 ? 0 : cx + 1;
  const int ys = cy == 0 ? L.ty - 1 : cy - 1, yn = cy == L.ty - 1 ? 0 : cy + 1;
  int tx = cx, ty = cy, off, row, col, p0, p1, p2;
  uint16_t kind = kPollWord;
  if (e < 2 * rw) {
    const bool below = e < rw;
    const int x = below ? e : e - rw;
    ty = below ? ys : yn;
    off = (below ? res_off_n(L) : res_off_s(L)) + x;
    row = below ? -1 : h;
    col = k16 ? 2 * x : x;
    p0 = below ? 2 : 4, p1 = below ? 5 : 7, p2 = below ? 6 : 8;
    // The last pair of an odd row ends in its first cell: the second is the ring's corner.
    if (k16 && col + 1 >= w) kind = kPollLow;
  } else if (e < 2 * (rw + h)) {
    e -= 2 * rw;
    const bool left = e < h;
    row = left ? e : e - h;
    tx = left ? xw : xe;
    off = (left ? res_off_e(L) : res_off_w(L)) + row;
    col = left ? -1 : w;
    p0 = left ? 1 : 3, p1 = left ? 5 : 6, p2 = left ? 8 : 7;
    if (k16) kind = kPollLow;
  } else {
    e -= 2 * (rw + h);
    const bool left = e == 0 || e == 2, below = e < 2;
    tx = left ? xw : xe;
    ty = below ? ys : yn;
    const int x = left ? L.width(xw, nx) - 1 : 0;
    off = (below ? res_off_n(L) : res_off_s(L)) + (k16 ? x >> 1 : x);
    row = below ? -1 : h;
    col = left ? -1 : w;
    p0 = -1, p1 = e == 0 ? 5 : (e == 3 ? 7 : -1), p2 = e == 1 ? 6 : (e == 2 ? 8 : -1);
    if (k16) kind = (x & 1) ? kPollHigh : kPollLow;
  }
  const int at = (row + 1) * rs + c0 + col;
  PollEntry q;
  q.src = static_cast<uint32_t>((ty * L.tx + tx) * L.words() + off);
  q.d[0] = p0 < 0 ? kPollSkip : static_cast<uint16_t>(p0 * PS + at);
  q.d[1] = p1 < 0 ? kPollSkip : static_cast<uint16_t>(p1 * PS + at);
  q.d[2] = p2 < 0 ? kPollSkip : static_cast<uint16_t>(p2 * PS + at);
  q.kind = kind;
  return q;
}

// A block's work items, one warp each. The tile's edge is a thin frame around the rest, so that
// its values leave early and travel while the interior is computed: first the bottom and top rows
// in groups of 32 cells (or pairs), then the first and last column (pair column) of the rows
// between with lanes along y, then the interior in groups of 32 along x.
template <int kElem>
struct ResItems {
  static constexpr int LC = kElem == 2 ? 2 : 1, GW = 32 * LC;
  int w, h, inner;          // inner: rows between the bottom and the top one
  int xlast;                // first cell of the last column (pair)
  int row_groups, in_groups;  // groups of a full row, of an interior row (cells LC .. xlast - 1)
  int row_items, col_items, total;
  RES_HD ResItems(int w_, int h_) : w(w_), h(h_) {
    inner = h > 2 ? h - 2 : 0;
    xlast = (w - 1) / LC * LC;
    row_groups = (w + GW - 1) / GW;
    in_groups = xlast > LC ? (xlast - LC + GW - 1) / GW : 0;
    row_items = (h > 1 ? 2 : 1) * row_groups;
    col_items = ((xlast > 0 ? 2 : 1) * inner + 31) / 32;
    total = row_items + col_items + inner * in_groups;
  }
  // Item e for one lane: its cell (or the pair's first), and whether it is on the frame; x < 0
  // where the lane has none.
  RES_HD void cell(int e, int lane, int& x, int& y, bool& frame) const {
    frame = true;
    if (e < row_items) {
      const bool top = e >= row_groups;
      y = top ? h - 1 : 0;
      x = (top ? e - row_groups : e) * GW + LC * lane;
      if (x >= w) x = -1;
      return;
    }
    e -= row_items;
    if (e < col_items) {
      const int t = 32 * e + lane;
      const bool second = t >= inner;
      y = 1 + (second ? t - inner : t);
      x = !second ? 0 : (t < 2 * inner && xlast > 0 ? xlast : -1);
      return;
    }
    e -= col_items;
    frame = false;
    const int r = e / in_groups;
    y = 1 + r;
    x = LC + (e - r * in_groups) * GW + LC * lane;
    if (x >= xlast) x = -1;
  }
};

// The cut into tx columns and ty bands, with tx = 0 where it is not one: columns are whole groups
// wide (mask words, 128-byte lines), the outlet's column nx - 2 shares its tile, and a tile's
// planes and tables fit the block.
template <int kElem>
inline ResLayout resident_cut(int nx, int ny, int tx, int ty, bool open_x) {
  constexpr int GW = kElem == 2 ? 64 : 32;
  ResLayout L;
  int w = (nx + tx - 1) / tx;
  if (tx > 1) w = (w + GW - 1) / GW * GW;
  const int h = (ny + ty - 1) / ty;
  if ((nx + w - 1) / w != tx || w > 4095 || h > 4095) return L;  // (fewer columns give the same cut)
  if (open_x && nx - (tx - 1) * w < 2) return L;
  if (static_cast<long long>(h + 2) * res_stride<kElem>(w) > kResPlaneBytes / kElem) return L;
  if (ResItems<kElem>(w, h).total > kResMaxItems || (h + 2) * ((w + 2 + 31) / 32 + 1) > kResMaxMask ||
      res_polls<kElem>(w, h) > kResMaxWords)
    return L;
  L.tx = tx;
  L.ty = ty;
  L.w = w;
  L.base = ny / ty;
  L.extra = ny % ty;
  L.hs = h;
  L.ws = res_row_words<kElem>(w);
  return L;
}
// Items of a cut's largest tile.
template <int kElem>
inline int resident_items(const ResLayout& L) {
  return ResItems<kElem>(L.w, L.hs).total;
}

// Cuts an nx x ny grid into at most `blocks` tiles for kElem-byte storage: the fewest rounds of
// the block's `warps` warps over its items, then the fewest items, then the shortest edge. Closed
// grids of at most 128 columns are cut into bands of one or two whole rows instead, 3/5 as many as
// rows, where that is at most half the blocks: as fast for one solver (us a step, spread over the
// SMs against bands: FP32 53 x 31 1.29 / 1.28, 64 x 64 1.29 / 1.29, 128 x 66 1.31 / 1.31, 120 x 40
// 1.33 / 1.26, 75 x 81 1.31 / 1.39; FP16 128 x 66 1.49 / 1.47, 40 x 60 1.50 / 1.53), and it leaves
// SMs to other solvers, whose resident launches otherwise wait (eight at once, us a step of all,
// spread / bands / one launch per step: FP32 53 x 31 5.2 / 1.4 / 3.6, 128 x 66 10.6 / 3.6 / 3.8; FP16
// 128 x 66 12.0 / 4.0 / 5.0). Bands cost more for one solver with wider rows (FP16 256 x 120 1.50 /
// 1.58) and open ends (FP32 128 x 66 1.35 / 1.42), which stay spread, as do grids that need the SMs
// (256 x 256: one solver 1.64 us on 152 SMs, 2.08 on 76; eight 12.9 / 8.4, one launch per step 9.4).
// Returns a layout with tx = 0 when no cut fits.
template <int kElem>
inline ResLayout resident_layout(int nx, int ny, int blocks, int warps, bool open_x) {
  const int bands = static_cast<int>((3LL * ny + 4) / 5);
  if (!open_x && nx <= 128 && 2 * bands <= blocks) {
    const ResLayout L = resident_cut<kElem>(nx, ny, 1, bands, false);
    if (L.tx) return L;
  }
  ResLayout best;
  long long best_cost = -1;
  for (int tx = 1; tx <= blocks; ++tx) {
    const ResLayout L = resident_cut<kElem>(nx, ny, tx, std::min(ny, blocks / tx), open_x);
    if (L.tx == 0) continue;
    const long long items = resident_items<kElem>(L), rounds = (items + warps - 1) / warps;
    const long long cost = (rounds * 1024 + items) * 65536 + res_polls<kElem>(L.w, L.hs);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = L;
    }
  }
  return best;
}

// The closed cut of an nx x ny grid with the fewest tiles of at most `items` items each (tx = 0:
// none), for ensembles that share the blocks.
template <int kElem>
inline ResLayout resident_layout_for(int nx, int ny, int items) {
  ResLayout best;
  const int max_tx = (nx + 31) / 32;
  for (int tx = 1; tx <= max_tx; ++tx) {
    // The tallest band that keeps the tile within `items` and the plane (both grow with it).
    int lo = 0, hi = ny;
    while (lo < hi) {
      const int h = (lo + hi + 1) / 2, ty = (ny + h - 1) / h;
      const ResLayout L = resident_cut<kElem>(nx, ny, tx, ty, false);
      if (L.tx && resident_items<kElem>(L) <= items)
        lo = h;
      else
        hi = h - 1;
    }
    if (lo == 0) continue;
    const ResLayout L = resident_cut<kElem>(nx, ny, tx, (ny + lo - 1) / lo, false);
    if (L.tx && (best.tx == 0 || L.tx * L.ty < best.tx * best.ty)) best = L;
  }
  return best;
}

}  // namespace lbm_b200
