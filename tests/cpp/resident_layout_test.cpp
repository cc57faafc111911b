// Host model of the resident kernel's exchange (csrc/resident_layout.h): for many grids, every
// tile fills its buffer with slot numbers, writes its edges to its outbox as the kernel's
// res_publish does, and reads its poll list back; then every population a cell
// pulls must be the slot the periodic lattice says, every item's cells must be covered once, and
// every index must stay inside its array. Exit status 0 when all hold.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "resident_layout.h"

using namespace lbm_b200;

namespace {

constexpr int CX[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
constexpr int CY[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};

long fails = 0;
#define CHECK(c, ...)                       \
  do {                                      \
    if (!(c)) {                             \
      if (fails < 10) std::printf(__VA_ARGS__); \
      ++fails;                              \
    }                                       \
  } while (0)

// Slot of population i of cell (x, y): nonzero, below 2^31 (a 16-bit "cell" carries it whole: the
// model moves slots, not bits, and splits pairs itself).
using Slot = long long;

template <int E>
void grid(int nx, int ny, int blocks, bool open, const ResLayout& L) {
  constexpr int PS = kResPlaneBytes / E, LC = E == 2 ? 2 : 1;
  if (L.tx == 0) return;
  CHECK(L.tx * L.ty <= blocks, "%dx%d: %d x %d tiles\n", nx, ny, L.tx, L.ty);
  const int tiles = L.tx * L.ty, nw = L.words(), c0 = res_col0<E>();
  struct Word {
    Slot lo[3] = {-1, -1, -1}, hi[3] = {-1, -1, -1};
  };
  std::vector<Word> box(static_cast<size_t>(tiles) * nw);
  std::vector<std::vector<Slot>> buf(tiles, std::vector<Slot>(9 * PS, -1));
  auto slot = [&](int i, int x, int y) { return (static_cast<Slot>(i) * ny + y) * nx + x + 1; };
  long cells = 0;
  for (int t = 0; t < tiles; ++t) {
    const int cx = t % L.tx, cy = t / L.tx, w = L.width(cx, nx), h = L.height(cy);
    const int x0 = cx * L.w, y0 = L.row0(cy), rs = res_stride<E>(w);
    const ResItems<E> items(w, h);
    CHECK(w >= 1 && h >= 1 && w <= L.w && h <= L.hs, "%dx%d tile %d: %d x %d\n", nx, ny, t, w, h);
    CHECK(!open || cx != L.tx - 1 || w >= 2, "%dx%d: outlet tile of one column\n", nx, ny);
    CHECK((h + 2) * rs <= PS && items.total <= kResMaxItems, "%dx%d tile %d does not fit\n", nx, ny, t);
    CHECK((h + 2) * ((w + 2 + 31) / 32 + 1) <= kResMaxMask && res_polls<E>(w, h) <= kResMaxWords, "%dx%d tables\n", nx, ny);
    auto& b = buf[t];
    std::vector<int> seen(w * h, 0);
    auto put = [&](int off, const int (&planes)[3], auto&& val, int k, bool both) {
      CHECK(off >= 0 && off < nw, "%dx%d tile %d: outbox word %d of %d\n", nx, ny, t, off, nw);
      if (off < 0 || off >= nw) return;
      Word v;
      for (int j = 0; j < 3; ++j) {
        v.lo[j] = val(planes[j], k);
        v.hi[j] = both ? val(planes[j], 1) : Slot(0);
      }
      box[static_cast<size_t>(t) * nw + off] = v;
    };
    for (int e = 0; e < items.total; ++e) {
      for (int lane = 0; lane < 32; ++lane) {
        int x, y;
        bool frame;
        items.cell(e, lane, x, y, frame);
        if (x < 0) continue;
        CHECK(x % LC == 0 && x < w && y >= 0 && y < h, "%dx%d tile %d: item %d cell %d,%d\n", nx, ny, t, e, x, y);
        const bool edge = y == 0 || y == h - 1 || x == 0 || x + LC >= w;
        CHECK(edge == frame, "%dx%d tile %d: cell %d,%d frame %d\n", nx, ny, t, x, y, frame);
        auto val = [&](int i, int k) { return x + k < w ? slot(i, x0 + x + k, y0 + y) : Slot(0); };
        for (int k = 0; k < LC && x + k < w; ++k) {
          ++seen[y * w + x + k];
          for (int i = 0; i < 9; ++i) b[i * PS + (y + 1) * rs + c0 + x + k] = val(i, k);
        }
        const int xr = x / LC;
        const int pn[3] = {2, 5, 6}, ps[3] = {4, 7, 8}, pe[3] = {1, 5, 8}, pw[3] = {3, 6, 7};
        if (y == h - 1) put(res_off_n(L) + xr, pn, val, 0, LC == 2);
        if (y == 0) put(res_off_s(L) + xr, ps, val, 0, LC == 2);
        if (LC == 2 ? (x | 1) >= w - 1 : x == w - 1)
          put(res_off_e(L) + y, pe, val, LC == 2 ? (w - 1) & 1 : 0, false);
        if (x == 0) put(res_off_w(L) + y, pw, val, 0, false);
      }
    }
    for (int s : seen) CHECK(s == 1, "%dx%d tile %d: a cell is taken %d times\n", nx, ny, t, s);
    cells += w * h;
  }
  CHECK(cells == static_cast<long>(nx) * ny, "%dx%d: %ld cells\n", nx, ny, cells);
  for (int t = 0; t < tiles; ++t) {
    const int cx = t % L.tx, cy = t / L.tx, w = L.width(cx, nx), h = L.height(cy);
    const int x0 = cx * L.w, y0 = L.row0(cy), rs = res_stride<E>(w);
    auto& b = buf[t];
    for (int e = 0; e < res_polls<E>(w, h); ++e) {
      const PollEntry q = res_poll_entry<E>(L, nx, cx, cy, w, h, e);
      CHECK(q.src < box.size(), "%dx%d: poll of word %u\n", nx, ny, q.src);
      if (q.src >= box.size()) continue;
      const Word v = box[q.src];
      for (int j = 0; j < 3; ++j) {
        if (q.d[j] == kPollSkip) continue;
        const uint32_t d = q.d[j];
        const bool pair = E == 2 && q.kind == kPollWord;
        CHECK(d + pair < static_cast<uint32_t>(9 * PS) && (!pair || d % 2 == 0), "%dx%d: ring slot %u\n", nx, ny, d);
        CHECK(v.lo[j] >= 0 && b[d] == -1, "%dx%d tile %d: word never written, or a slot written twice\n", nx, ny, t);
        b[d] = q.kind == kPollHigh ? v.hi[j] : v.lo[j];
        if (pair) {
          CHECK(b[d + 1] == -1, "%dx%d tile %d: a pair overwrites its neighbour\n", nx, ny, t);
          b[d + 1] = v.hi[j];
        }
      }
    }
    for (int y = 0; y < h; ++y)
      for (int x = 0; x < w; ++x)
        for (int i = 0; i < 9; ++i) {
          const int gx = (x0 + x - CX[i] + nx) % nx, gy = (y0 + y - CY[i] + ny) % ny;
          const Slot got = b[i * PS + (y + 1 - CY[i]) * rs + c0 + x - CX[i]];
          CHECK(got == slot(i, gx, gy), "%dx%d tile %d cell %d,%d dir %d: %lld\n", nx, ny, t, x, y, i, got);
        }
  }
}

template <int E>
long sweep() {
  long n = 0;
  for (int blocks : {1, 7, 152})
    for (bool open : {false, true}) {
      for (int nx : {1, 2, 3, 33, 64, 65, 66, 128, 300, 1021, 1025})
        for (int ny : {1, 2, 3, 7, 31, 152, 153, 320, 700}) {
          if (open && nx < 3) continue;
          grid<E>(nx, ny, blocks, open, resident_layout<E>(nx, ny, blocks, 28, open));
          if (!open && blocks == 152) {
            const int items = 5 + (nx * 7 + ny) % 60;
            const ResLayout L = resident_layout_for<E>(nx, ny, items);
            CHECK(L.tx == 0 || resident_items<E>(L) <= items, "%dx%d: more than %d items\n", nx, ny, items);
            grid<E>(nx, ny, 1 << 20, false, L);
          }
          ++n;
        }
    }
  return n;
}

}  // namespace

int main() {
  const long n = sweep<4>() + sweep<2>();
  std::printf("%ld grids, %ld failures\n", n, fails);
  return fails == 0 ? 0 : 1;
}
