// Resident stream-collide: many steps per launch with the state in shared memory.
//
// A grid small enough for the SMs' shared memory is cut into tiles, one per SM (one block each,
// launched cooperatively so that all are resident). A block loads its tile's pull state once,
// takes `steps` steps between two shared-memory buffers, exchanging only the populations that
// cross its edges with its neighbours, and writes the tile back. Against one launch per step
// (about 3 us of launch chain and pipeline fill whatever the size) a step costs its collisions
// plus one exchange.
//
//   * A buffer holds, per plane, rows -1 .. h of columns -1 .. w: the tile and the ring of cells
//     around it that its pull reads. Periodic wrap is then no special case (the ring comes from
//     the tile on the other side, possibly the tile itself).
//   * Exchange: every population leaving through an edge is written by the thread that computed
//     it, with the other two of its cell that cross that edge, as one 16-byte word {three values,
//     tag} to the tile's outbox in global memory (L2); the neighbour's threads poll the word
//     itself until it carries the state's tag (the step number of the whole run, unique over
//     launches). The 16-byte access is single-copy atomic, so the tag vouches for its values and
//     no fence or flag round trip is needed: one store and one load
//     latency per step. Outboxes alternate between two parities: a tile overwrites parity q's
//     words for state t + 2 only after it has read all eight neighbours' words of state t + 1,
//     which they wrote after reading state t.
//   * A block's work is a list of items (32 cells, or 32 pairs with 16-bit storage, per warp): the
//     tile's one-cell frame first, so that the words travel while the interior is computed. One
//     barrier per step.
//   * Bound by: instruction issue on the larger tiles (FP32 1024 x 256: 2.5 us a step, 57 items of
//     about 270 instructions on 32 warps, 80 % issue between the barriers), the exchange's
//     latency (about 0.9 us) on small ones (128 x 66: 1.3 us). us a step at 400 steps a call, with one
//     launch per step in parentheses: FP32 53 x 31 1.3 (2.7), 256^2 1.7 (3.1), 512^2 2.3 (4.9), 1024
//     x 256 2.4 (4.8), 1000 x 320 open 2.9 (6.6); FP16 128 x 66 1.5 (3.7), 512^2 2.4 (4.2), 1021 x 700
//     3.4 (7.9).
//   * Measured and left out: words of one value and an 8-byte tag (three times the stores and
//     polls: 1024 x 256 2.90 us); whole-row items for the frame, which hold up the words until most
//     of the tile is done (512^2 3.16 against 2.47 us); two FP32 cells per lane in packed
//     instructions (27 % fewer instructions, but 92 registers leave 20 warps for 29 items:
//     1024 x 256 2.66 us, 512^2 2.70 us).
//   * Waits are bounded (kResidentPolls; a kernel argument, so that a test can shorten them); a wait
//     that runs out sets the error flag and ends the block, and its neighbours' waits run out in
//     turn.
#pragma once

#include "resident_layout.h"
#include "step_ring.cuh"

namespace lbm_b200 {

constexpr unsigned kResidentPolls = 1u << 22;  // about 2 s
// Shortest run that takes a resident launch (solver.cu has the figures), and steps per launch (a
// few tens of milliseconds).
constexpr int kResidentMinSteps = 4, kResidentSteps = 8192;

// One outbox word {v0, v1, v2, tag}: a 16-byte access that is single-copy atomic.
struct alignas(16) LLWord {
  uint32_t v[3], tag;
};
__device__ __forceinline__ void ll_store(LLWord* p, uint32_t a, uint32_t b, uint32_t c, uint32_t tag) {
  asm volatile(
      "{\n"
      ".reg .b64 lo, hi;\n"
      ".reg .b128 q;\n"
      "mov.b64 lo, {%1, %2};\n"
      "mov.b64 hi, {%3, %4};\n"
      "mov.b128 q, {lo, hi};\n"
      "st.relaxed.gpu.global.b128 [%0], q;\n"
      "}\n" ::"l"(p),
      "r"(a), "r"(b), "r"(c), "r"(tag)
      : "memory");
}
__device__ __forceinline__ LLWord ll_load(const LLWord* p) {
  LLWord w;
  asm volatile(
      "{\n"
      ".reg .b64 lo, hi;\n"
      ".reg .b128 q;\n"
      "ld.relaxed.gpu.global.b128 q, [%4];\n"
      "mov.b128 {lo, hi}, q;\n"
      "mov.b64 {%0, %1}, lo;\n"
      "mov.b64 {%2, %3}, hi;\n"
      "}\n"
      : "=r"(w.v[0]), "=r"(w.v[1]), "=r"(w.v[2]), "=r"(w.tag)
      : "l"(p)
      : "memory");
  return w;
}

// Edge values of cell x, y of a w x h tile, a frame cell, into its outbox. 32-bit values: the
// cell's populations, or with 16-bit storage the pair's (cells x, x + 1, low cell first).
__device__ __forceinline__ uint32_t res_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t res_bits(uint32_t v) { return v; }
template <bool kPair, class V>
__device__ __forceinline__ void res_publish(const V (&v)[kQ], const ResLayout& L, LLWord* ob, uint32_t tag, int x,
                                            int y, int w, int h) {
  const int xr = kPair ? x >> 1 : x;
  if (y == h - 1) ll_store(ob + res_off_n(L) + xr, res_bits(v[2]), res_bits(v[5]), res_bits(v[6]), tag);
  if (y == 0) ll_store(ob + res_off_s(L) + xr, res_bits(v[4]), res_bits(v[7]), res_bits(v[8]), tag);
  if (kPair ? (x | 1) >= w - 1 : x == w - 1) {
    const int sh = kPair ? ((w - 1) & 1) * 16 : 0;  // cell w - 1 in the low half
    ll_store(ob + res_off_e(L) + y, res_bits(v[1]) >> sh, res_bits(v[5]) >> sh, res_bits(v[8]) >> sh, tag);
  }
  if (x == 0) ll_store(ob + res_off_w(L) + y, res_bits(v[3]), res_bits(v[6]), res_bits(v[7]), tag);
}

// The lane's cell (or pair) of an item: gathers from `cur`, collides, stores to `nxt` and, for a
// frame cell (publish), to the outbox. x, y: tile coordinates of the cell (or of the pair's
// first); solids: the item holds or touches solid cells.
template <class ST, class Phys, bool kOpen, int kForce>
__device__ __forceinline__ void res_cell(const StepArgs<ST, Phys>& p, const ST* cur, ST* nxt, int rs,
                                         const uint32_t* mask, int mw, const ResLayout& L, LLWord* ob, uint32_t tag,
                                         bool solids, bool publish, uint32_t rkey, int x, int y, int w, int h, int gx,
                                         int gy) {
  constexpr int PS = kResPlaneBytes / static_cast<int>(sizeof(ST));
  const int o = (y + 1) * rs + res_col0<static_cast<int>(sizeof(ST))>() + x;
  const int nx = p.g.nx;
  const ST* c = cur + o;
  uint32_t nm = 0, n0 = 0, np = 0;
  if constexpr (sizeof(ST) == 4) {
    float v[kQ];
#pragma unroll
    for (int i = 0; i < kQ; ++i) v[i] = c[i * PS - dir_cy(i) * rs - dir_cx(i)];
    if (solids) {
      const uint32_t* m = mask + y * mw + (x >> 5);
      const int sh = x & 31;
      nm = __funnelshift_r(m[0], m[1], sh) & 7u;
      n0 = __funnelshift_r(m[mw], m[mw + 1], sh) & 7u;
      np = __funnelshift_r(m[2 * mw], m[2 * mw + 1], sh) & 7u;
      if (!(n0 & 2u)) {
#pragma unroll
        for (int i = 1; i < kQ; ++i) {
          const uint32_t b = dir_cy(i) == 1 ? nm : (dir_cy(i) == -1 ? np : n0);
          if ((b >> (1 - dir_cx(i))) & 1u) v[i] = c[dir_opp(i) * PS];
        }
      }
    }
    if (kOpen) {
      if (gx == 0) {
        v[1] = p.eq_in[1];
        v[5] = p.eq_in[5];
        v[8] = p.eq_in[8];
      }
      if (gx == nx - 1) {
#pragma unroll
        for (int i = 1; i < kQ; ++i) {
          if (dir_cx(i) != -1) continue;
          const uint32_t b = dir_cy(i) == 1 ? nm : (dir_cy(i) == -1 ? np : n0);
          if (!((b >> 1) & 1u))
            v[i] = c[i * PS - dir_cy(i) * rs];
          else  // nothing from a solid cell nx - 2
            v[i] = (n0 & 1u) ? 0.0f : c[dir_opp(i) * PS - 1];
        }
      }
    }
    float out[kQ];
    collide_exact_kind<typename Phys::Arith, kForce>(v, p.k, out);
    ST* d = nxt + o;
#pragma unroll
    for (int i = 0; i < kQ; ++i) d[i * PS] = out[i];
    if (publish) res_publish<false>(out, L, ob, tag, x, y, w, h);
  } else {
    float2 v[kQ];
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
      const uint32_t* r = reinterpret_cast<const uint32_t*>(c + i * PS - dir_cy(i) * rs);
      const uint32_t own = r[0];
      uint32_t raw = own;
      if (dir_cx(i) == 1) raw = __byte_perm(r[-1], own, 0x5432);
      if (dir_cx(i) == -1) raw = __byte_perm(own, r[1], 0x5432);
      v[i] = widen_pair<ST>(raw);
    }
    if (solids) {
      const uint32_t* m = mask + y * mw + (x >> 5);
      const int sh = x & 31;
      nm = __funnelshift_r(m[0], m[1], sh) & 15u;
      n0 = __funnelshift_r(m[mw], m[mw + 1], sh) & 15u;
      np = __funnelshift_r(m[2 * mw], m[2 * mw + 1], sh) & 15u;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if ((n0 >> (1 + k)) & 1u) continue;
#pragma unroll
        for (int i = 1; i < kQ; ++i) {
          const uint32_t b = dir_cy(i) == 1 ? nm : (dir_cy(i) == -1 ? np : n0);
          if ((b >> (1 + k - dir_cx(i))) & 1u) {
            const float t = widen<ST>(c[dir_opp(i) * PS + k]);
            if (k == 0) v[i].x = t; else v[i].y = t;
          }
        }
      }
    }
    if (kOpen) {
      if (gx == 0) {
        v[1].x = p.eq_in[1];
        v[5].x = p.eq_in[5];
        v[8].x = p.eq_in[8];
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (gx + k != nx - 1) continue;
#pragma unroll
        for (int i = 1; i < kQ; ++i) {
          if (dir_cx(i) != -1) continue;
          const uint32_t b = dir_cy(i) == 1 ? nm : (dir_cy(i) == -1 ? np : n0);
          float t = 0.0f;
          if (!((b >> (1 + k)) & 1u))
            t = widen<ST>(c[i * PS - dir_cy(i) * rs + k]);
          else if (!((n0 >> k) & 1u))
            t = widen<ST>(c[dir_opp(i) * PS + k - 1]);
          if (k == 0) v[i].x = t; else v[i].y = t;
        }
      }
    }
    float2 out[kQ];
    collide_fast_t<FastF32x2, kForce>(v, p.k, out);
    const uint32_t ph = sr_pair_hash(p.key_base + static_cast<long long>(gy) * p.g.pitch + gx, rkey);
    uint32_t q[kQ];
#pragma unroll
    for (int i = 0; i < kQ; ++i) q[i] = encode_pair_sr<ST>(out[i].x, out[i].y, i, ph);
    ST* d = nxt + o;
    if (x + 1 < w) {
#pragma unroll
      for (int i = 0; i < kQ; ++i) *reinterpret_cast<uint32_t*>(d + i * PS) = q[i];
    } else {  // the second cell's slot belongs to the ring
#pragma unroll
      for (int i = 0; i < kQ; ++i) *reinterpret_cast<uint16_t*>(d + i * PS) = static_cast<uint16_t>(q[i]);
    }
    if (publish) res_publish<true>(q, L, ob, tag, x, y, w, h);
  }
}

// A block's item table: first cell of a row or interior item, or the index of a column item,
// | row << 12 | flags (solid: a cell of the item, or a neighbour of one, is solid).
constexpr uint32_t kItemSolid = 1u << 24, kItemFrame = 1u << 25, kItemColumn = 1u << 26;

// Threads of a resident block: what the collision's registers allow (64 for the exact FP32 one,
// 72 for the 16-bit one).
template <class ST>
__host__ __device__ constexpr int res_threads() {
  return sizeof(ST) == 2 ? 896 : 1024;
}

// The steps of tile `tile` of the grid p, cut as L. The state is read from and written back to
// p.dst (p.src is unused); `outboxes` are the grid's, of both parities; *tag_ctr numbers the states
// (it only ever grows, see above), *p.step_ctr keys the stochastic rounding. A word is looked at
// `polls_limit` times at most.
template <class ST, class Phys, bool kOpen, int kForce>
__device__ __forceinline__ void resident_body(unsigned char* smem, const StepArgs<ST, Phys>& p, const ResLayout& L,
                                              int tile, int steps, LLWord* outboxes, const uint32_t* tag_ctr,
                                              int* err, unsigned polls_limit) {
  constexpr int PS = kResPlaneBytes / static_cast<int>(sizeof(ST));
  constexpr int LC = sizeof(ST) == 2 ? 2 : 1, kThreads = res_threads<ST>();
  ST* buf0 = reinterpret_cast<ST*>(smem);
  ST* buf1 = buf0 + 9 * PS;
  PollEntry* polls = reinterpret_cast<PollEntry*>(smem + 18 * static_cast<size_t>(kResPlaneBytes));
  uint32_t* mask = reinterpret_cast<uint32_t*>(polls + kResMaxWords);
  uint32_t* table = mask + kResMaxMask;  // per item, see kItem*

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nx = p.g.nx, ny = p.g.ny;
  const int cy = tile / L.tx, cx = tile - cy * L.tx;
  const int w = L.width(cx, nx), h = L.height(cy), x0 = cx * L.w, y0 = L.row0(cy);
  const int rs = res_stride<static_cast<int>(sizeof(ST))>(w), c0 = res_col0<static_cast<int>(sizeof(ST))>();
  const ResItems<static_cast<int>(sizeof(ST))> items(w, h);
  const int nitems = items.total, npolls = res_polls<static_cast<int>(sizeof(ST))>(w, h);
  const int mw = (w + 2 + 31) / 32 + 1;
  const long long per_parity = static_cast<long long>(L.words()) * L.tx * L.ty;
  // Tags start at 1: outboxes are created as zeros.
  const uint32_t t0 = __ldg(tag_ctr) + 1u, step0 = sizeof(ST) == 2 ? __ldg(p.step_ctr) : 0u;

  // Tables: mask bits (bit j of a row: cell x0 - 1 + j; rows -1 .. h), poll list, items.
  for (int k = tid; k < (h + 2) * mw; k += kThreads) {
    const int r = k / mw, q = k - r * mw;
    int y = y0 - 1 + r;
    y = y < 0 ? ny - 1 : (y >= ny ? 0 : y);
    mask[k] = mask_window(p.mask + static_cast<size_t>(y) * p.g.mask_words, x0 + 32 * q);
  }
  for (int e = tid; e < npolls; e += kThreads) polls[e] = res_poll_entry<static_cast<int>(sizeof(ST))>(L, nx, cx, cy, w, h, e);
  __syncthreads();
  for (int e = warp; e < nitems; e += kThreads / 32) {
    int x, y;
    bool frame;
    items.cell(e, lane, x, y, frame);
    uint32_t any = 0;
    if (x >= 0)
      for (int r = 0; r < 3; ++r) {
        const uint32_t* m = mask + (y + r) * mw + (x >> 5);
        any |= __funnelshift_r(m[0], m[1], x & 31) & (LC == 2 ? 15u : 7u);
      }
    any = __any_sync(0xffffffffu, any != 0u);
    const bool col = frame && e >= items.row_items;
    if (lane == 0)
      table[e] = static_cast<uint32_t>(col ? e - items.row_items : x) | (static_cast<uint32_t>(y) << 12) |
                 (any ? kItemSolid : 0u) | (frame ? kItemFrame : 0u) | (col ? kItemColumn : 0u);
  }
  // The tile's state, and its edges for the neighbours (state t0).
  {
    const ST* g = p.dst + static_cast<long long>(y0) * p.g.pitch + x0;
    const int n = w * h;
    for (int k = tid; k < n; k += kThreads) {
      const int y = k / w, x = k - y * w;
#pragma unroll
      for (int i = 0; i < kQ; ++i)
        buf0[i * PS + (y + 1) * rs + c0 + x] = __ldcg(g + i * p.g.plane + static_cast<long long>(y) * p.g.pitch + x);
    }
  }
  __syncthreads();
  LLWord* mine = outboxes + static_cast<long long>(tile) * L.words();
  {
    LLWord* ob = mine + (t0 & 1u) * per_parity;
    for (int e = warp; e < items.row_items + items.col_items; e += kThreads / 32) {
      int x, y;
      bool frame;
      items.cell(e, lane, x, y, frame);
      if (x < 0) continue;
      const ST* c = buf0 + (y + 1) * rs + c0 + x;
      using V = std::conditional_t<LC == 1, float, uint32_t>;
      V v[kQ];
#pragma unroll
      for (int i = 0; i < kQ; ++i) v[i] = *reinterpret_cast<const V*>(c + i * PS);
      res_publish<LC == 2>(v, L, ob, t0, x, y, w, h);
    }
  }
  ST *cur = buf0, *nxt = buf1;
  bool ok = true;
  // Reads the ring of the state with tag `tag` into `b`. The last warps, which have the fewest
  // items, take the first words.
  auto receive = [&](ST* b, uint32_t tag) {
    const LLWord* from = outboxes + (tag & 1u) * per_parity;
    for (int e = kThreads - 1 - tid; e < npolls; e += kThreads) {
      const PollEntry q = polls[e];
      LLWord v = ll_load(from + q.src);
      for (unsigned n = 1; v.tag != tag; ++n) {
        if (n >= polls_limit) {
          atomicExch(err, 1);
          ok = false;
          break;
        }
        v = ll_load(from + q.src);
      }
      if (!ok) break;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (q.d[j] == kPollSkip) continue;
        ST* d = b + q.d[j];
        if (LC == 1 || q.kind == kPollWord)
          *reinterpret_cast<uint32_t*>(d) = v.v[j];
        else
          *reinterpret_cast<uint16_t*>(d) = static_cast<uint16_t>(q.kind == kPollHigh ? v.v[j] >> 16 : v.v[j]);
      }
    }
  };
  receive(cur, t0);
  bool dead = __syncthreads_or(!ok);
  for (int k = 0; k < steps && !dead; ++k) {
    const uint32_t tag = t0 + static_cast<uint32_t>(k) + 1u;
    const bool more = k + 1 < steps;
    LLWord* ob = mine + (tag & 1u) * per_parity;
    const uint32_t rkey = sizeof(ST) == 2 ? sr_step_key(step0 + static_cast<uint32_t>(k)) : 0u;
    for (int e = warp; e < nitems; e += kThreads / 32) {
      const uint32_t it = table[e];
      int x = static_cast<int>(it & 0xfffu) + LC * lane, y = static_cast<int>((it >> 12) & 0xfffu);
      bool mine_cell = x < ((it & kItemFrame) ? w : items.xlast);
      if (it & kItemColumn) {
        const int t = 32 * static_cast<int>(it & 0xfffu) + lane;
        const bool second = t >= items.inner;
        y = 1 + (second ? t - items.inner : t);
        x = second ? items.xlast : 0;
        mine_cell = t < (items.xlast > 0 ? 2 : 1) * items.inner;
      }
      if (mine_cell)
        res_cell<ST, Phys, kOpen, kForce>(p, cur, nxt, rs, mask, mw, L, ob, tag, (it & kItemSolid) != 0u,
                                          more && (it & kItemFrame) != 0u, rkey, x, y, w, h, x0 + x, y0 + y);
    }
    if (more) receive(nxt, tag);
    dead = __syncthreads_or(!ok);
    ST* s = cur;
    cur = nxt;
    nxt = s;
  }
  {
    ST* g = p.dst + static_cast<long long>(y0) * p.g.pitch + x0;
    const int n = w * h;
    for (int k = tid; k < n; k += kThreads) {
      const int y = k / w, x = k - y * w;
#pragma unroll
      for (int i = 0; i < kQ; ++i)
        g[i * p.g.plane + static_cast<long long>(y) * p.g.pitch + x] = cur[i * PS + (y + 1) * rs + c0 + x];
    }
  }
}

// One grid: block k has tile k.
template <class ST, class Phys, bool kOpen, int kForce>
__global__ void __launch_bounds__(res_threads<ST>(), 1)
    resident_step_kernel(const StepArgs<ST, Phys> p, const ResLayout L, int steps, LLWord* outboxes, int* err,
                         unsigned polls_limit) {
  extern __shared__ __align__(128) unsigned char smem[];
  resident_body<ST, Phys, kOpen, kForce>(smem, p, L, static_cast<int>(blockIdx.x), steps, outboxes, p.step_ctr, err,
                                         polls_limit);
}

}  // namespace lbm_b200
