// Single-grid solver: device memory, launches and the C ABI of include/lbm_b200.h.
//
// Host code of this file is compiled with -ffp-contract=off: the per-launch constants (omega,
// the force prefactor, the inlet and initial equilibria) are computed here in the solver
// precision with the reference's expressions, and must round exactly as the reference's host
// code does (src/v3_cuda_opt/solver_v3.cu:194-226,252-253).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "aux_kernels.cuh"
#include "host_access.h"
#include "lbm_b200.h"
#include "solver_internal.h"
#include "step_kernel.cuh"
#include "step_async.cuh"
#include "step_resident.cuh"
#include "step_ring.cuh"
#include "step_tma.cuh"
#include "stream_sms.h"
#include "forms.cuh"

using namespace lbm_b200;

namespace {

int set_error(lbm_solver* s, int code, const std::string& msg) {
  if (s) s->err = msg;
  return code;
}

int cuda_fail(lbm_solver* s, cudaError_t e, const char* what) {
  cudaGetLastError();  // clear a sticky launch error so that later calls can report their own
  const int code = e == cudaErrorMemoryAllocation ? LBM_ERR_OUT_OF_MEMORY : LBM_ERR_CUDA;
  return set_error(s, code, std::string(what) + ": " + cudaGetErrorString(e));
}

#define LBM_CUDA(s, call)                                   \
  do {                                                      \
    const cudaError_t lbm_e_ = (call);                      \
    if (lbm_e_ != cudaSuccess) return cuda_fail(s, lbm_e_, #call); \
  } while (0)

int grid_for_cells(const lbm_solver* s, long long n, int block) {
  const long long want = (n + block - 1) / block;
  return static_cast<int>(std::max<long long>(1, std::min<long long>(want, 32LL * s->sm_count)));
}

template <class ST>
Eq9<typename StoreTraits<ST>::T> inlet_eq(const lbm_solver* s) {
  using T = typename StoreTraits<ST>::T;
  if (!s->open_x) return Eq9<T>{};
  return host_equilibrium<T>(T(1), T(s->u_in), T(0));
}

// The inlet equilibrium in the step kernels' compute representation (16-bit forms: scaled).
template <class ST>
Eq9<typename StoreTraits<ST>::T> step_inlet_eq(const lbm_solver* s) {
  Eq9<typename StoreTraits<ST>::T> e = inlet_eq<ST>(s);
  if (sizeof(ST) == 2)
    for (int i = 0; i < kQ; ++i) e.v[i] *= s->sc.enc[i];
  return e;
}

// Physics of a launch: the scalar form, or (kPacked) its two-cells-per-instruction twin.
template <class ST, bool kPacked>
using PhysOf = std::conditional_t<kPacked, typename Form<ST>::PackedPhys, typename Form<ST>::Phys>;

template <class ST, bool kOpen, int kVariant, class Phys = typename Form<ST>::Phys>
int launch_steps_t(lbm_solver* s, int steps) {
  using T = typename StoreTraits<ST>::T;
  constexpr int G = StoreTraits<ST>::kVec;
  StepArgs<ST, Phys> a{};
  a.mask = s->mask_d;
  a.g = s->g;
  a.cpr = (s->nx + 32 * G - 1) / (32 * G);
  a.items = s->ny * a.cpr;
  a.k = Form<ST>::consts(s->tau, s->fx, s->fy);
  const Eq9<T> e = step_inlet_eq<ST>(s);
  for (int i = 0; i < kQ; ++i) a.eq_in[i] = e.v[i];
  a.sc = s->sc;
  const auto kernel = pull_step_kernel<ST, Phys, kOpen, kVariant>;
  // FP64 with integer multiplications holds 141 registers: blocks of half the size let 12 warps
  // reside instead of 8 and even out the last wave (300 x 300: 2.60k MLUPS with 256 threads).
  constexpr bool kInt = std::is_same_v<Phys, F64IntPhys>;
  const int block = kInt && !s->block_set ? 128 : s->block;
  int grid = s->grid;
  if (grid <= 0) {
    int per_sm = 0;
    LBM_CUDA(s, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0));
    if (kInt) per_sm = kF64GridPerSm;
    const int warps_per_block = block / 32;
    const int need = (a.items + warps_per_block - 1) / warps_per_block;
    grid = std::max(1, std::min(need, std::max(1, per_sm) * s->sm_count));
  }
  s->last_block = block;
  s->last_grid = grid;
  for (int k = 0; k < steps; ++k) {
    a.src = static_cast<const ST*>(s->buf[s->cur]);
    a.dst = static_cast<ST*>(s->buf[s->cur ^ 1]);
    a.step_ctr = s->step_ctr;
    a.step_off = static_cast<uint32_t>(k);
    LBM_CUDA(s, launch_dependent(kernel, dim3(grid), dim3(block), 0, s->stream, a));
    s->cur ^= 1;
  }
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

// Warp-specialised bulk-copy step (step_tma.cuh) with kStages ring stages.
template <class ST, bool kOpen, int kStages, bool kPacked = false>
int launch_tma_t(lbm_solver* s, int steps) {
  using Phys = PhysOf<ST, kPacked>;
  using T = typename StoreTraits<ST>::T;
  using S = TmaShape<ST>;
  StepArgs<ST, Phys> a{};
  a.mask = s->mask_d;
  a.g = s->g;
  a.cpr = (s->nx + 32 * S::G - 1) / (32 * S::G);
  a.items = s->ny * a.cpr;
  a.k = Form<ST>::consts(s->tau, s->fx, s->fy);
  const Eq9<T> e = step_inlet_eq<ST>(s);
  for (int i = 0; i < kQ; ++i) a.eq_in[i] = e.v[i];
  a.sc = s->sc;
  const int tpr = (s->nx + S::TW - 1) / S::TW;
  const int tiles = tpr * s->ny;
  const auto kernel = tma_step_kernel<ST, Phys, kOpen, kStages>;
  const size_t smem = tma_smem_bytes<ST>(kStages);
  LBM_CUDA(s, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem)));
  int grid = s->grid;
  if (grid <= 0) {
    int per_sm = 0;
    LBM_CUDA(s, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTmaThreads, smem));
    grid = std::max(1, std::min(tiles, std::max(1, per_sm) * s->sm_count));
  }
  s->last_grid = grid;
  for (int k = 0; k < steps; ++k) {
    a.src = static_cast<const ST*>(s->buf[s->cur]);
    a.dst = static_cast<ST*>(s->buf[s->cur ^ 1]);
    a.step_ctr = s->step_ctr;
    a.step_off = static_cast<uint32_t>(k);
    LBM_CUDA(s, launch_dependent(kernel, dim3(grid), dim3(kTmaThreads), smem, s->stream, a, tpr, tiles,
                                 s->err_flag));
    s->cur ^= 1;
  }
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

// Per-warp asynchronous-copy pipeline (step_async.cuh), kDepth chunks per warp, 4 warps per block.
template <class ST, bool kOpen, int kDepth, bool kPacked = true>
int launch_async_t(lbm_solver* s, int steps) {
  using Phys = PhysOf<ST, kPacked>;
  using T = typename StoreTraits<ST>::T;
  constexpr int G = StoreTraits<ST>::kVec;
  constexpr int kBlock = 128;
  StepArgs<ST, Phys> a{};
  a.mask = s->mask_d;
  a.g = s->g;
  a.cpr = (s->nx + 32 * G - 1) / (32 * G);
  a.items = s->ny * a.cpr;
  a.k = Form<ST>::consts(s->tau, s->fx, s->fy);
  const Eq9<T> e = step_inlet_eq<ST>(s);
  for (int i = 0; i < kQ; ++i) a.eq_in[i] = e.v[i];
  a.sc = s->sc;
  const auto kernel = async_step_kernel<ST, Phys, kOpen, kDepth>;
  const size_t smem = async_smem_bytes<ST>(kDepth, kBlock / 32);
  LBM_CUDA(s, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem)));
  int grid = s->grid;
  if (grid <= 0) {
    int per_sm = 0;
    LBM_CUDA(s, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, smem));
    const int need = (a.items + kBlock / 32 - 1) / (kBlock / 32);
    grid = std::max(1, std::min(need, std::max(1, per_sm) * s->sm_count));
  }
  s->last_grid = grid;
  for (int k = 0; k < steps; ++k) {
    a.src = static_cast<const ST*>(s->buf[s->cur]);
    a.dst = static_cast<ST*>(s->buf[s->cur ^ 1]);
    a.step_ctr = s->step_ctr;
    a.step_off = static_cast<uint32_t>(k);
    LBM_CUDA(s, launch_dependent(kernel, dim3(grid), dim3(kBlock), smem, s->stream, a));
    s->cur ^= 1;
  }
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

// Warp-specialised ring with one cell (plain FP32 / FP64) or one pair of cells (16-bit storage)
// per lane (step_ring.cuh). kMaxBlocks > 0 caps the resident blocks per SM (by the shared memory
// a block asks for): past the bytes in flight that cover the latency, more of them only queue in
// front of HBM and cost bandwidth (FP32, 4096^2, variant 12: 87.1k MLUPS at the 3 blocks per SM
// it was tuned for, 78.5k at the 4 its 56 registers allow).
template <class ST, bool kOpen, int kW, int kC, int kStages, int kMinBlocks, int kMaxBlocks = 0,
          class Phys = typename Form<ST>::Phys>
int launch_ring_t(lbm_solver* s, int steps) {
  {
    using T = typename StoreTraits<ST>::T;
    using S = RingShape<ST, kW, kC>;
    StepArgs<ST, Phys> a{};
    a.mask = s->mask_d;
    a.g = s->g;
    a.k = Form<ST>::consts(s->tau, s->fx, s->fy);
    const Eq9<T> e = step_inlet_eq<ST>(s);
    for (int i = 0; i < kQ; ++i) a.eq_in[i] = e.v[i];
    a.sc = s->sc;
    const int tpr = (s->nx + S::TW - 1) / S::TW;
    const int tiles = tpr * s->ny;
    const auto kernel = ring_step_kernel<ST, Phys, kOpen, kW, kC, kStages, kMinBlocks>;
    size_t smem = ring_smem_bytes<S>(kStages);
    if (kMaxBlocks > 0) smem = std::max(smem, smem_for_blocks(kMaxBlocks));
    LBM_CUDA(s, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(smem)));
    int grid = s->grid;
    if (grid <= 0) {
      int per_sm = 0;
      LBM_CUDA(s, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, S::kThreads, smem));
      if (sizeof(ST) == 8) per_sm = kF64GridPerSm;
      grid = std::max(1, std::min(tiles, std::max(1, per_sm) * s->sm_count));
    }
    s->last_grid = grid;
    for (int k = 0; k < steps; ++k) {
      a.src = static_cast<const ST*>(s->buf[s->cur]);
      a.dst = static_cast<ST*>(s->buf[s->cur ^ 1]);
      a.step_ctr = s->step_ctr;
      a.step_off = static_cast<uint32_t>(k);
      // Odd steps (by buffer parity) walk the tiles backwards: they start on the rows the
      // previous step wrote last.
      LBM_CUDA(s, launch_dependent(kernel, dim3(grid), dim3(S::kThreads), smem, s->stream, a, tpr, tiles, 0,
                                   s->cur, s->err_flag));
      s->cur ^= 1;
    }
    LBM_CUDA(s, cudaGetLastError());
    return LBM_OK;
  }
}

// Variant of the automatic choice: the ring with 4 consumer warps, 2 passes (256-cell
// tiles), 2 stages and 5 resident blocks per SM, for plain FP32 on large grids. With fewer
// instructions per cell the earlier choice (12, then 63 registers and so 3 blocks) drains its
// stages faster and keeps too many bytes queued: 4096^2 MLUPS by shape and blocks per SM: 12
// with 4 blocks 78.5k, 3 blocks 87.1k, 2 blocks 86.4k; 15 with 3 blocks 89.7k; this one with 4 / 5 / 6
// blocks 89.0k / 90.9k / 79k (3000 x 5000: 87.9k / 91.1k / 79k; 2048^2: 85.4k / 87.8k / 84.6k).
// The largest grids take 3 stages and 3 blocks (28): 8192^2 91.1k against 87.9k, 8192 x 6000 91.8k /
// 88.8k, 10000 x 7000 89.1k / 85.2k, 16384 x 4096 91.3k / 88.3k; 6000^2 84.7k / 91.2k, 5000^2 89.7k /
// 90.6k.
constexpr int kVariantF32Large = 23, kVariantF32Largest = 28;

// Variant of the automatic choice: 20 with at most 2 resident blocks per SM, for 16-bit
// storage on grids of at least 2^23 cells.
constexpr int kVariant16Large = 27;

// Variants of the automatic choice in FP64: ring and direct kernel with integer multiplications.
constexpr int kVariantF64Ring = 25, kVariantF64Direct = 26;

// Variant number of resident launches (step_resident.cuh). A launch loads and stores the
// state and has no dependent-launch overlap, so short runs stay with the step kernels (us a step,
// resident against them, runs of 4 / 16 / 400 steps: FP32 128 x 66 3.2 / 1.8 / 1.3 against 3.6 /
// 3.0 / 2.9; 1024 x 256 5.3 / 3.0 / 2.3 against 6.0 / 5.2 / 4.8; FP16 1021 x 700 7.0 / 4.3 / 3.4
// against 8.9 / 8.2 / 7.9): from four steps on every size that fits is faster resident, for one
// solver at a time (resident_layout.h has several).
constexpr int kVariantResident = 24;

// Automatic kernel choice (variant < 0), from a sweep of every variant on one GB300 (channel,
// best of 3 runs, MLUPS): plain FP32: 256^2 v19 20.8k (v0 19.8k), 512^2 / 1024x256 v17 51.9k /
// 51.7k (v12 47.4k / 46.2k), 1024^2 v17 83.9k (v12 81.7k), 2048^2 v12 86.2k, 4096^2 v12 90.6k;
// 16-bit storage: 256^2 v19 20.2k (v0 13.5k), 512^2 v19 61.2k, 1024^2 v19 114.5k (v17 108.6k,
// v20 91.1k: its 2048-cell tiles are half empty on 1024-cell rows), 2048^2 v20 157.1k (v17
// 143.0k), 4096^2 v20 168.7k (v17 159.3k). With the one-instruction stochastic conversion
// (fewer instructions per cell) the 16-bit sweep moved on the largest grids (walled channel,
// seeded state, best of 3): 2048^2 v20 170.6k (v17 149.7k), 4096^2 v20 169.5k (v17 169.0k,
// v22 170.3k), 8192^2 v17 175.7k (v20 168.9k). Variant 20 kept to 2 resident blocks per SM (27)
// queues less in front of HBM: 4096^2 174.2k, 6144 x 4096 176.2k (v17 171.9k), 8192^2 178.1k; at
// 2048^2, whose states lie half in L2, 153.8k against 171k with 3 blocks.
// Rows narrower than 256 cells take the
// direct kernel (0), whose 128-cell chunks leave fewer lanes idle than the rings' wide tiles
// (FP64 on 100 x 2000: the ring 12 reached 1.0k MLUPS with a fifth of its lanes busy). FP64
// takes kernels of its own, with the multiplications on the integer units (mul64.h), bound by the
// FP64 pipe's additions: the ring with 256-cell tiles, 4 stages, 3 blocks per SM (MLUPS at
// 1024 x 512: 2.56k with the hardware's multiplications and the resident grid, 3.07k with the
// shorter collision and the larger grid, 4.72k with integer multiplications; 2048^2 4.90k; with
// no force 6.02k), the direct kernel where the row's 256-cell tiles are less than 95 % full.
template <class ST>
int auto_variant(const lbm_solver* s) {
  using S = RingShape<ST, 8, 2>;
  const long long cells = static_cast<long long>(s->nx) * s->ny;
  if (s->nx < 256) return sizeof(ST) == 8 ? kVariantF64Direct : 0;
  if (sizeof(ST) == 8) {
    const int tw = S::TW / 2;
    return 20LL * s->nx < 19LL * ((s->nx + tw - 1) / tw * tw) ? kVariantF64Direct : kVariantF64Ring;
  }
  if (sizeof(ST) == 2) {
    if (cells < (2LL << 20)) return 19;
    if (cells < (4LL << 20) || !wide_tiles16(s->nx)) return 17;
    return cells < (8LL << 20) ? 20 : kVariant16Large;
  }
  if (cells < (2LL << 20)) return cells < (1LL << 17) ? 19 : 17;
  return cells < (44LL << 20) ? kVariantF32Large : kVariantF32Largest;
}

template <class ST, bool kOpen>
int launch_steps_o(lbm_solver* s, int steps) {
  s->last_variant = s->variant >= 0 && s->variant != kVariantResident ? s->variant : auto_variant<ST>(s);
  s->last_block = 0;
  // The automatic choice's own kernels, of one storage form each.
  if constexpr (sizeof(ST) == 8) {
    if (s->last_variant == kVariantF64Ring) return launch_ring_t<ST, kOpen, 8, 1, 4, 3, 0, F64IntPhys>(s, steps);
    if (s->last_variant == kVariantF64Direct) return launch_steps_t<ST, kOpen, 0, F64IntPhys>(s, steps);
  } else if constexpr (sizeof(ST) == 4) {
    if (s->last_variant == kVariantF32Large) return launch_ring_t<ST, kOpen, 4, 2, 2, 5, 5>(s, steps);
    if (s->last_variant == kVariantF32Largest) return launch_ring_t<ST, kOpen, 4, 2, 3, 1, 3>(s, steps);
  } else {
    if (s->last_variant == kVariant16Large) return launch_ring_t<ST, kOpen, 8, 4, 2, 2, 2>(s, steps);
  }
  switch (s->last_variant) {
    case 1: return launch_steps_t<ST, kOpen, 1>(s, steps);
    case 2: return launch_steps_t<ST, kOpen, 2>(s, steps);
    case 3: return launch_steps_t<ST, kOpen, 3>(s, steps);
    case 4: return launch_tma_t<ST, kOpen, 2>(s, steps);
    case 5: return launch_tma_t<ST, kOpen, 3>(s, steps);
    case 6: return launch_tma_t<ST, kOpen, 4>(s, steps);
    case 7: return launch_tma_t<ST, kOpen, 2, true>(s, steps);
    case 8: return launch_steps_t<ST, kOpen, 0, PhysOf<ST, true>>(s, steps);
    case 9: return launch_async_t<ST, kOpen, 2>(s, steps);
    case 10: return launch_async_t<ST, kOpen, 3>(s, steps);
    case 11: return launch_async_t<ST, kOpen, 4>(s, steps);
    case 12: return launch_ring_t<ST, kOpen, 8, 2, 2, 1, sizeof(ST) == 4 ? 3 : 0>(s, steps);
    case 13: return launch_ring_t<ST, kOpen, 8, 2, 3, 1, sizeof(ST) == 4 ? 3 : 0>(s, steps);
    case 14: return launch_ring_t<ST, kOpen, 8, 2, 2, 4>(s, steps);
    case 15: return launch_ring_t<ST, kOpen, 4, 2, 3, 1>(s, steps);
    case 16: return launch_ring_t<ST, kOpen, 4, 2, 3, 7>(s, steps);
    case 17: return launch_ring_t<ST, kOpen, 8, 2, 2, 3>(s, steps);
    case 18: return launch_ring_t<ST, kOpen, 8, 2, 3, 3>(s, steps);
    case 19: return launch_ring_t<ST, kOpen, 8, 1, 4, 3>(s, steps);
    case 20: return launch_ring_t<ST, kOpen, 8, 4, 2, 2>(s, steps);
    case 21: return launch_ring_t<ST, kOpen, 4, 4, 2, 5>(s, steps);
    case 22: return launch_ring_t<ST, kOpen, 8, 4, 3, 2>(s, steps);
    default: return launch_steps_t<ST, kOpen, 0>(s, steps);
  }
}

// A cooperative launch that was refused because its blocks cannot all be resident: nothing of it
// ran, and the step kernels take the steps.
constexpr int kRefused = -1;

// Resident launches: the whole run of `steps` in cooperative launches of at most
// kResidentSteps steps each, the state in the blocks' shared memory meanwhile. kRefused with the
// first of them.
template <class ST, bool kOpen, int kForce>
int launch_resident_t(lbm_solver* s, int steps) {
  using Phys = typename Form<ST>::Phys;
  using T = typename StoreTraits<ST>::T;
  StepArgs<ST, Phys> a{};
  a.mask = s->mask_d;
  a.g = s->g;
  a.k = Form<ST>::consts(s->tau, s->fx, s->fy);
  const Eq9<T> e = step_inlet_eq<ST>(s);
  for (int i = 0; i < kQ; ++i) a.eq_in[i] = e.v[i];
  a.sc = s->sc;
  a.dst = static_cast<ST*>(s->buf[s->cur]);
  a.step_ctr = s->step_ctr;
  const auto kernel = resident_step_kernel<ST, Phys, kOpen, kForce>;
  LBM_CUDA(s, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(kResSmemBytes)));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(s->res.tx * s->res.ty);
  cfg.blockDim = dim3(res_threads<ST>());
  cfg.dynamicSmemBytes = kResSmemBytes;
  cfg.stream = s->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  for (int done = 0; done < steps;) {
    const int n = std::min(steps - done, kResidentSteps);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a, s->res, n, static_cast<LLWord*>(s->outbox), s->err_flag,
                                             g_resident_polls.load());
    if (e == cudaErrorCooperativeLaunchTooLarge && done == 0) {
      cudaGetLastError();
      return kRefused;
    }
    LBM_CUDA(s, e);
    LBM_CUDA(s, launch_dependent(counter_add_dep_kernel, dim3(1), dim3(1), 0, s->stream, s->step_ctr,
                                 static_cast<uint32_t>(n)));
    s->enqueued += 2;
    done += n;
  }
  s->last_grid = s->res.tx * s->res.ty;
  s->last_variant = kVariantResident;
  s->last_block = 0;
  return LBM_OK;
}

template <class ST>
int launch_resident(lbm_solver* s, int steps) {
  int rc = kRefused;
  if constexpr (sizeof(ST) != 8)
    with_force(Form<ST>::consts(s->tau, s->fx, s->fy).force, [&](auto kind) {
      constexpr int K = decltype(kind)::value;
      rc = s->open_x ? launch_resident_t<ST, true, K>(s, steps) : launch_resident_t<ST, false, K>(s, steps);
    });
  return rc;
}

// Do the step kernels' launch sequences end with a counter update?
bool counts_steps(const lbm_solver* s) { return s->elem == 2; }

// Runs of at least kResidentMinSteps steps take resident launches where the grid fits, its blocks
// the SMs that the stream may use, and the caller has not chosen a kernel.
bool use_resident(const lbm_solver* s, int steps) {
  return s->res.tx > 0 && (s->variant < 0 || s->variant == kVariantResident) && s->grid == 0 && s->block == kStepThreads && steps >= kResidentMinSteps &&
         s->res.tx * s->res.ty <= stream_sm_count(s->stream, s->sm_count);
}

template <class ST>
int launch_steps(lbm_solver* s, int steps) {
  const int rc = s->open_x ? launch_steps_o<ST, true>(s, steps) : launch_steps_o<ST, false>(s, steps);
  if (rc) return rc;
  // The counter keys the rounding of the 16-bit forms (and numbers resident states, whose launches
  // advance it themselves): FP32 and FP64 steps go without the update.
  if (counts_steps(s))
    LBM_CUDA(s, launch_dependent(counter_add_dep_kernel, dim3(1), dim3(1), 0, s->stream, s->step_ctr,
                                 static_cast<uint32_t>(steps)));
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

// The current state from a uniform equilibrium, or from v0-layout populations that kernels can
// address.
template <class ST>
int set_equilibrium_t(lbm_solver* s, Eq9<typename StoreTraits<ST>::T> eq) {
  const long long n = static_cast<long long>(s->nx) * s->ny;
  set_state_kernel<ST><<<grid_for_cells(s, n, 256), 256, 0, s->stream>>>(static_cast<ST*>(s->buf[s->cur]), s->mask_d,
                                                                         s->g, nullptr, eq, s->sc);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}
template <class ST>
int set_state_t(lbm_solver* s, const void* aos) {
  using T = typename StoreTraits<ST>::T;
  const long long n = static_cast<long long>(s->nx) * s->ny;
  scatter_state_kernel<ST><<<grid_for_cells(s, n, kGetThreads), kGetThreads, 0, s->stream>>>(
      static_cast<ST*>(s->buf[s->cur]), s->mask_d, s->g, static_cast<const T*>(aos), s->sc);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int get_state_t(lbm_solver* s, void* aos_dev) {
  using T = typename StoreTraits<ST>::T;
  const long long n = static_cast<long long>(s->nx) * s->ny;
  get_state_kernel<ST><<<grid_for_cells(s, n, 256), kGetThreads, 0, s->stream>>>(
      static_cast<const ST*>(s->buf[s->cur]), s->mask_d, s->g, inlet_eq<ST>(s), s->sc,
      static_cast<T*>(aos_dev), 0, s->ny);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int moments_t(lbm_solver* s, void* rho, void* ux, void* uy) {
  using A = typename Form<ST>::A;
  using T = typename A::T;
  const long long n = static_cast<long long>(s->nx) * s->ny;
  const T hfx = T(0.5) * T(s->fx), hfy = T(0.5) * T(s->fy);
  moments_kernel<ST, A><<<grid_for_cells(s, n, 256), 256, 0, s->stream>>>(
      static_cast<const ST*>(s->buf[s->cur]), s->mask_d, s->g, inlet_eq<ST>(s), s->sc, hfx, hfy,
      static_cast<T*>(rho), static_cast<T*>(ux), static_cast<T*>(uy), 0, s->ny);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int mass_t(lbm_solver* s, const void* state, double* partials, int blocks, double* out) {
  mass_partial_kernel<ST><<<blocks, kReduceThreads, 0, s->stream>>>(
      static_cast<const ST*>(state), s->mask_d, s->g, inlet_eq<ST>(s), s->sc, partials);
  mass_final_kernel<<<1, kReduceThreads, 0, s->stream>>>(partials, blocks,
                                                         static_cast<double>(s->fluid), out);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int finite_t(lbm_solver* s, int* flag) {
  const long long n = static_cast<long long>(s->nx) * s->ny;
  finite_kernel<ST><<<grid_for_cells(s, n, 256), 256, 0, s->stream>>>(
      static_cast<const ST*>(s->buf[s->cur]), s->mask_d, s->g, s->sc, flag);
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int body_force_t(lbm_solver* s, double* out) {
  const uint32_t* body = s->body_d ? s->body_d : s->mask_d;
  // Only cells next to the body feel it: scan the box around it (the whole grid without one).
  int box[4] = {0, 0, s->nx, s->ny};
  if (s->body_d) std::copy(s->body_box, s->body_box + 4, box);
  const long long n = static_cast<long long>(box[2]) * box[3];
  const int blocks =
      static_cast<int>(std::max<long long>(1, std::min<long long>(s->red_blocks, (n + kReduceThreads - 1) / kReduceThreads)));
  body_force_partial_kernel<ST><<<blocks, kReduceThreads, 0, s->stream>>>(
      static_cast<const ST*>(s->buf[s->cur]), s->mask_d, body, s->g, s->sc, box[0], box[1], box[2], box[3],
      s->force_red);
  LBM_CUDA(s, launch_dependent(pair_final_kernel, dim3(1), dim3(kReduceThreads), 0, s->stream,
                               static_cast<const double*>(s->force_red), blocks, out));
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

template <class ST>
int probe_t(lbm_solver* s, int x, int y, void* out) {
  using T = typename StoreTraits<ST>::T;
  probe_kernel<ST><<<1, 32, 0, s->stream>>>(static_cast<const ST*>(s->buf[s->cur]), s->mask_d,
                                            s->g, inlet_eq<ST>(s), s->sc, x, y,
                                            static_cast<T*>(out));
  LBM_CUDA(s, cudaGetLastError());
  return LBM_OK;
}

// Dispatch on the storage form (one code path per form, no fallback).
#define LBM_DISPATCH(s, fn, ...)                                       \
  switch ((s)->precision) {                                           \
    case LBM_FP32: return fn<float>(__VA_ARGS__);                     \
    case LBM_FP64: return fn<double>(__VA_ARGS__);                    \
    case LBM_FP16_STORE: return fn<__half>(__VA_ARGS__);              \
    case LBM_BF16_STORE: return fn<__nv_bfloat16>(__VA_ARGS__);       \
    default: return set_error(s, LBM_ERR_INVALID_ARG, "bad precision"); \
  }

template <class ST>
int init_eq_t(lbm_solver* s, double rho0, double ux0, double uy0) {
  using T = typename StoreTraits<ST>::T;
  return set_equilibrium_t<ST>(s, host_equilibrium<T>(T(rho0), T(ux0), T(uy0)));
}

int ensure_stage(lbm_solver* s, size_t bytes) {
  if (s->stage_bytes >= bytes) return LBM_OK;
  if (s->stage) {
    LBM_CUDA(s, cudaStreamSynchronize(s->stream));
    cudaFree(s->stage);
    s->stage = nullptr;
    s->stage_bytes = 0;
  }
  LBM_CUDA(s, cudaMalloc(&s->stage, bytes));
  s->stage_bytes = bytes;
  return LBM_OK;
}

// The cut of the grid for resident launches: tx = 0 where the grid does not fit.
ResLayout plan_resident(const lbm_solver* s, bool open_x) {
  if (s->elem == 4) return resident_layout<4>(s->nx, s->ny, s->sm_count, res_threads<float>() / 32, open_x);
  if (s->elem == 2) return resident_layout<2>(s->nx, s->ny, s->sm_count, res_threads<__half>() / 32, open_x);
  return ResLayout{};
}
size_t outbox_bytes(const ResLayout& L) { return 2 * static_cast<size_t>(L.words()) * L.tx * L.ty * sizeof(LLWord); }

int check(const lbm_solver* s) { return s ? LBM_OK : LBM_ERR_INVALID_ARG; }

// Storage scales: 1 for the plain forms, kStoreScale16 (2^15) on every plane of the 16-bit forms
// (the largest stored magnitude 65504 / 2^15 ~ 2 bounds |g_i| = |f_i - w_i| of any state with
// 0 <= f_i <= 1, and values down to 2^-29 stay normal).
PlaneScales default_scales(int precision) {
  PlaneScales p{};
  const bool s16 = precision == LBM_FP16_STORE || precision == LBM_BF16_STORE;
  for (int i = 0; i < kQ; ++i) {
    p.enc[i] = s16 ? kStoreScale16 : 1.0f;
    p.dec[i] = s16 ? 1.0f / kStoreScale16 : 1.0f;
  }
  return p;
}

}  // namespace

// ----------------------------------------------------------------------------------------------
// Internal helpers shared with the other translation units
// ----------------------------------------------------------------------------------------------
namespace lbm_b200 {

std::atomic<unsigned> g_resident_polls{kResidentPolls};

int solver_launch(lbm_solver* s, int steps) { LBM_DISPATCH(s, launch_steps, s, steps); }
static int solver_launch_resident(lbm_solver* s, int steps) { LBM_DISPATCH(s, launch_resident, s, steps); }

void drop_step_graph(lbm_solver* s) {
  if (s->graph) cudaGraphExecDestroy(s->graph);
  s->graph = nullptr;
  s->graph_cur = -1;
}

// Captures kGraphSteps step launches (and the step-counter update) from the current buffer
// parity into a CUDA graph. kGraphSteps is even, so a replay leaves the parity unchanged. A
// capture that fails turns graphs off for this solver (direct launches give the same results).
int ensure_step_graph(lbm_solver* s) {
  if (s->graph && s->graph_cur == s->cur) return LBM_OK;
  drop_step_graph(s);
  const int cur0 = s->cur;
  cudaGraph_t g = nullptr;
  if (cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    cudaGetLastError();
    s->graphs = false;
    return LBM_OK;
  }
  const int rc = solver_launch(s, kGraphSteps);
  const cudaError_t e = cudaStreamEndCapture(s->stream, &g);
  s->cur = cur0;
  if (rc || e != cudaSuccess || !g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    s->graphs = false;
    return LBM_OK;
  }
  const cudaError_t ei = cudaGraphInstantiate(&s->graph, g, 0);
  cudaGraphDestroy(g);
  if (ei != cudaSuccess) {
    cudaGetLastError();
    s->graph = nullptr;
    s->graphs = false;
    return LBM_OK;
  }
  s->graph_cur = cur0;
  return LBM_OK;
}

// Steps: resident launches where they apply, else whole CUDA graphs of kGraphSteps launches for long
// runs on a non-default stream (no per-launch host overhead, which dominates small grids), direct
// launches for the remainder.
int solver_step_raw(lbm_solver* s, int steps) {
  if (use_resident(s, steps)) {
    const int rc = solver_launch_resident(s, steps);
    if (!rc) s->kernels += steps + 1;
    if (rc != kRefused) return rc;
  }
  if (s->graphs && s->stream != nullptr && steps >= kGraphSteps) {
    if (int rc = ensure_step_graph(s)) return rc;
    while (s->graph && steps >= kGraphSteps) {
      LBM_CUDA(s, cudaGraphLaunch(s->graph, s->stream));
      s->kernels += kGraphSteps + (counts_steps(s) ? 1 : 0);  // the graph's launches
      s->enqueued += kGraphSteps + (counts_steps(s) ? 1 : 0);
      steps -= kGraphSteps;
    }
  }
  if (steps <= 0) return LBM_OK;
  const int rc = solver_launch(s, steps);
  if (!rc) {
    s->kernels += steps + (counts_steps(s) ? 1 : 0);
    s->enqueued += steps + (counts_steps(s) ? 1 : 0);
  }
  return rc;
}

int solver_mass_into(lbm_solver* s, const void* state, double* partials, int blocks,
                     double* out) {
  LBM_DISPATCH(s, mass_t, s, state, partials, blocks, out);
}

void pack_mask(const uint8_t* solid, int nx, int ny, int mask_words, std::vector<uint32_t>& out) {
  out.assign(static_cast<size_t>(mask_words) * ny, 0xffffffffu);
  const int used = (nx + 2 + 31) / 32;  // words that hold cells or periodic neighbours
  for (int y = 0; y < ny; ++y) {
    uint32_t* row = out.data() + static_cast<size_t>(y) * mask_words;
    const uint8_t* src = solid + static_cast<size_t>(y) * nx;
    for (int q = 0; q < used; ++q) {
      const int x0 = 32 * q - 1;  // bit 0's cell
      uint32_t v = 0;
      if (x0 >= 0 && x0 + 32 <= nx) {
        for (int j = 0; j < 32; ++j) v |= static_cast<uint32_t>(src[x0 + j] != 0) << j;
      } else {
        for (int j = 0; j < 32; ++j) {
          const int x = x0 + j;
          const bool s = x < 0 ? src[nx - 1] != 0 : (x < nx ? src[x] != 0 : (x == nx ? src[0] != 0 : true));
          v |= static_cast<uint32_t>(s) << j;
        }
      }
      row[q] = v;
    }
  }
}

int element_bytes(int precision) {
  switch (precision) {
    case LBM_FP32: return 4;
    case LBM_FP64: return 8;
    case LBM_FP16_STORE:
    case LBM_BF16_STORE: return 2;
    default: return 0;
  }
}

}  // namespace lbm_b200

// ----------------------------------------------------------------------------------------------
// C ABI
// ----------------------------------------------------------------------------------------------
extern "C" {

const char* lbm_version(void) { return "lbm_b200 1.0 (sm_103a)"; }

int lbm_create(int nx, int ny, const uint8_t* solid, double tau, double fx, double fy,
               int precision, lbm_solver** out) {
  if (!out) return LBM_ERR_INVALID_ARG;
  *out = nullptr;
  const int elem = element_bytes(precision);
  if (nx < 1 || ny < 1 || !solid || elem == 0) return LBM_ERR_INVALID_ARG;
  // The reference compares tau in its own precision (solver_v3.cu:169-170).
  const bool tau_ok = precision == LBM_FP64 ? tau > 0.5 : static_cast<float>(tau) > 0.5f;
  if (!tau_ok || !std::isfinite(tau) || !std::isfinite(fx) || !std::isfinite(fy))
    return LBM_ERR_INVALID_ARG;
  if (static_cast<long long>(nx) * ny > (1LL << 31) - 1) return LBM_ERR_INVALID_ARG;

  lbm_solver* s = new (std::nothrow) lbm_solver();
  if (!s) return LBM_ERR_OUT_OF_MEMORY;
  s->nx = nx;
  s->ny = ny;
  s->precision = precision;
  s->elem = elem;
  s->vec = 16 / elem;
  s->host_elem = precision == LBM_FP64 ? 8 : 4;
  s->tau = tau;
  s->fx = fx;
  s->fy = fy;
  s->solid.assign(solid, solid + static_cast<size_t>(nx) * ny);
  for (uint8_t v : s->solid) s->fluid += v ? 0 : 1;
  s->sc = default_scales(precision);

  const int per_line = 128 / elem;
  const int pitch = (nx + per_line - 1) / per_line * per_line;
  s->g.nx = nx;
  s->g.ny = ny;
  s->g.pitch = pitch;
  s->g.mask_words = mask_row_words(nx);
  s->g.plane = static_cast<long long>(pitch) * ny;
  s->g.open_x = 0;

  auto fail = [&](int code) {
    lbm_destroy(s);
    return code;
  };
  cudaError_t e = cudaGetDevice(&s->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, s->device);
  if (e != cudaSuccess) return fail(LBM_ERR_CUDA);
  e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) return fail(LBM_ERR_CUDA);
  s->own_stream = true;
  e = cudaEventCreate(&s->ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev[1]);
  if (e != cudaSuccess) return fail(LBM_ERR_CUDA);

  const size_t state_bytes = static_cast<size_t>(kQ) * s->g.plane * elem + 256;
  // The outboxes of resident launches, for the closed cut and the open one, lie behind the second
  // state: one allocation and one memset (of zeros: words of no state) less per solver.
  int coop = 0, optin = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device);
  const size_t out_at = (state_bytes + 255) / 256 * 256;
  size_t out_bytes = 0;
  s->can_reside = coop && static_cast<size_t>(optin) >= kResSmemBytes;
  if (s->can_reside) {
    s->res = plan_resident(s, false);
    out_bytes = std::max(outbox_bytes(s->res), outbox_bytes(plan_resident(s, true)));
  }
  for (int b = 0; b < 2; ++b) {
    const size_t bytes = b == 1 && out_bytes ? out_at + out_bytes : state_bytes;
    e = cudaMalloc(&s->buf[b], bytes);
    if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? LBM_ERR_OUT_OF_MEMORY : LBM_ERR_CUDA);
    e = cudaMemsetAsync(s->buf[b], 0, bytes, s->stream);
    if (e != cudaSuccess) return fail(LBM_ERR_CUDA);
  }
  if (out_bytes) s->outbox = static_cast<char*>(s->buf[1]) + out_at;
  s->state_bytes = state_bytes;
  std::vector<uint32_t> words;
  pack_mask(solid, nx, ny, s->g.mask_words, words);
  e = cudaMalloc(&s->mask_d, words.size() * sizeof(uint32_t));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(s->mask_d, words.data(), words.size() * sizeof(uint32_t),
                        cudaMemcpyHostToDevice, s->stream);
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? LBM_ERR_OUT_OF_MEMORY : LBM_ERR_CUDA);
  s->red_blocks = 4 * s->sm_count;
  const size_t red_bytes = (s->red_blocks + 2) * sizeof(double) + 4 * sizeof(int);
  e = cudaMalloc(&s->red, red_bytes);
  if (e == cudaSuccess) e = cudaMemsetAsync(s->red, 0, red_bytes, s->stream);
  s->direct = host_memory_direct(s->device);
  s->err_flag = s->direct ? const_cast<int*>(&s->box.flag) : reinterpret_cast<int*>(s->red + s->red_blocks + 2) + 1;
  s->step_ctr = reinterpret_cast<uint32_t*>(s->red + s->red_blocks + 2) + 2;
  if (e != cudaSuccess) return fail(e == cudaErrorMemoryAllocation ? LBM_ERR_OUT_OF_MEMORY : LBM_ERR_CUDA);
  e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return fail(LBM_ERR_CUDA);
  *out = s;
  return LBM_OK;
}

int lbm_destroy(lbm_solver* s) {
  if (!s) return LBM_OK;
  if (s->stream) cudaStreamSynchronize(s->stream);
  for (void* p : s->buf) cudaFree(p);
  cudaFree(s->mask_d);
  lbm_b200::drop_step_graph(s);
  cudaFree(s->red);
  cudaFree(s->body_d);
  cudaFree(s->force_red);
  cudaFree(s->stage);
  for (cudaEvent_t ev : s->ev)
    if (ev) cudaEventDestroy(ev);
  if (s->own_stream && s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return LBM_OK;
}

const char* lbm_last_error(const lbm_solver* s) { return s ? s->err.c_str() : "null solver"; }

int lbm_set_stream(lbm_solver* s, void* stream) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  if (s->own_stream) cudaStreamDestroy(s->stream);
  s->own_stream = false;
  s->stream = static_cast<cudaStream_t>(stream);
  return LBM_OK;
}

int lbm_set_inflow_outflow(lbm_solver* s, double u_in) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  if (s->nx < 3 || !std::isfinite(u_in))
    return set_error(s, LBM_ERR_INVALID_ARG, "open boundaries need nx >= 3 and a finite u_in");
  s->open_x = true;
  s->u_in = u_in;
  s->g.open_x = 1;
  if (s->can_reside) s->res = plan_resident(s, true);
  lbm_b200::drop_step_graph(s);
  return LBM_OK;
}

int lbm_init_equilibrium(lbm_solver* s, double rho0, double ux0, double uy0) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  LBM_DISPATCH(s, init_eq_t, s, rho0, ux0, uy0);
}

int lbm_set_populations(lbm_solver* s, const void* s_host) {
  if (check(s) || !s_host) return set_error(s, LBM_ERR_INVALID_ARG, "null state");
  const size_t bytes = static_cast<size_t>(s->nx) * s->ny * kQ * s->host_elem;
  // The conversion reads host memory that kernels can address in place (each value once, in
  // contiguous runs), else a copy of it in device memory.
  const void* src = host_view(s_host, bytes, s->host_elem, s->direct, false);
  if (!src) {
    if (int rc = ensure_stage(s, bytes)) return rc;
    LBM_CUDA(s, cudaMemcpyAsync(s->stage, s_host, bytes, cudaMemcpyHostToDevice, s->stream));
    src = s->stage;
  }
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = set_state_t<float>(s, src); break;
    case LBM_FP64: rc = set_state_t<double>(s, src); break;
    case LBM_FP16_STORE: rc = set_state_t<__half>(s, src); break;
    case LBM_BF16_STORE: rc = set_state_t<__nv_bfloat16>(s, src); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));  // the host buffer may be reused on return
  return LBM_OK;
}

int lbm_step(lbm_solver* s, int steps) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  if (steps < 0) return set_error(s, LBM_ERR_INVALID_ARG, "steps must be >= 0");
  if (steps == 0) return LBM_OK;
  return lbm_b200::solver_step_raw(s, steps);
}

// Reads and clears the device error flag of the step kernels (a bounded wait that ran out).
static int check_step_flag(lbm_solver* s) {
  if (s->direct) {
    LBM_CUDA(s, cudaStreamSynchronize(s->stream));
    if (!s->box.flag) return LBM_OK;
    s->box.flag = 0;
    return set_error(s, LBM_ERR_TIMEOUT, kWaitMessage);
  }
  int flag = 0;
  LBM_CUDA(s, cudaMemcpyAsync(&flag, s->err_flag, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  if (flag) {
    LBM_CUDA(s, cudaMemsetAsync(s->err_flag, 0, sizeof(int), s->stream));
    LBM_CUDA(s, cudaStreamSynchronize(s->stream));
    return set_error(s, LBM_ERR_TIMEOUT, kWaitMessage);
  }
  return LBM_OK;
}

int lbm_synchronize(lbm_solver* s) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  return check_step_flag(s);
}

int lbm_run(lbm_solver* s, int steps) {
  if (int rc = lbm_step(s, steps)) return rc;
  return lbm_synchronize(s);
}

int lbm_kernel_launches(const lbm_solver* s, long long* count) {
  if (!s || !count) return LBM_ERR_INVALID_ARG;
  *count = s->kernels;
  return LBM_OK;
}

int lbm_enqueued_kernels(const lbm_solver* s, long long* count) {
  if (!s || !count) return LBM_ERR_INVALID_ARG;
  *count = s->enqueued;
  return LBM_OK;
}

int lbm_timed_run(lbm_solver* s, int steps, double* seconds) {
  if (check(s) || !seconds) return set_error(s, LBM_ERR_INVALID_ARG, "null argument");
  LBM_CUDA(s, cudaEventRecord(s->ev[0], s->stream));
  if (int rc = lbm_step(s, steps)) return rc;
  LBM_CUDA(s, cudaEventRecord(s->ev[1], s->stream));
  LBM_CUDA(s, cudaEventSynchronize(s->ev[1]));
  float ms = 0.f;
  LBM_CUDA(s, cudaEventElapsedTime(&ms, s->ev[0], s->ev[1]));
  *seconds = static_cast<double>(ms) * 1e-3;
  return check_step_flag(s);
}

int lbm_get_populations(lbm_solver* s, void* s_host) {
  if (check(s) || !s_host) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  const size_t bytes = static_cast<size_t>(s->nx) * s->ny * kQ * s->host_elem;
  // Host output that kernels can address: the gather kernel writes it in place; else through
  // device memory.
  void* dst = host_view(s_host, bytes, s->host_elem, s->direct, true);
  if (!dst) {
    if (int rc = ensure_stage(s, bytes)) return rc;
    dst = s->stage;
  }
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = get_state_t<float>(s, dst); break;
    case LBM_FP64: rc = get_state_t<double>(s, dst); break;
    case LBM_FP16_STORE: rc = get_state_t<__half>(s, dst); break;
    case LBM_BF16_STORE: rc = get_state_t<__nv_bfloat16>(s, dst); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  if (dst == s->stage)
    LBM_CUDA(s, cudaMemcpyAsync(s_host, s->stage, bytes, cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  return LBM_OK;
}

int lbm_macroscopic(lbm_solver* s, void* rho, void* ux, void* uy) {
  if (check(s) || !rho || !ux || !uy) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  const size_t n = static_cast<size_t>(s->nx) * s->ny;
  const size_t plane = n * s->host_elem;
  // Host outputs that kernels can address (all three): the moment kernel writes them in place;
  // else through device memory.
  void* mr = host_view(rho, plane, s->host_elem, s->direct, true);
  void* mu = mr ? host_view(ux, plane, s->host_elem, s->direct, true) : nullptr;
  void* mv = mu ? host_view(uy, plane, s->host_elem, s->direct, true) : nullptr;
  const bool direct = mr && mu && mv;
  char* d = nullptr;
  if (!direct) {
    if (int rc = ensure_stage(s, std::max(3 * plane, n * kQ * s->host_elem))) return rc;
    d = static_cast<char*>(s->stage);
    mr = d;
    mu = d + plane;
    mv = d + 2 * plane;
  }
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = moments_t<float>(s, mr, mu, mv); break;
    case LBM_FP64: rc = moments_t<double>(s, mr, mu, mv); break;
    case LBM_FP16_STORE: rc = moments_t<__half>(s, mr, mu, mv); break;
    case LBM_BF16_STORE: rc = moments_t<__nv_bfloat16>(s, mr, mu, mv); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  if (!direct) {
    LBM_CUDA(s, cudaMemcpyAsync(rho, d, plane, cudaMemcpyDeviceToHost, s->stream));
    LBM_CUDA(s, cudaMemcpyAsync(ux, d + plane, plane, cudaMemcpyDeviceToHost, s->stream));
    LBM_CUDA(s, cudaMemcpyAsync(uy, d + 2 * plane, plane, cudaMemcpyDeviceToHost, s->stream));
  }
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  return LBM_OK;
}

int lbm_total_mass(lbm_solver* s, double* mass) {
  if (check(s) || !mass) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  double* out = s->direct ? s->box.out : s->red + s->red_blocks;
  if (int rc = lbm_b200::solver_mass_into(s, s->buf[s->cur], s->red, s->red_blocks, out)) return rc;
  if (s->direct) {
    LBM_CUDA(s, cudaStreamSynchronize(s->stream));
    *mass = s->box.out[0];
    return LBM_OK;
  }
  LBM_CUDA(s, cudaMemcpyAsync(mass, out, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  return LBM_OK;
}

int lbm_populations_at(lbm_solver* s, int x, int y, void* out9) {
  if (check(s) || !out9) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  if (x < 0 || x >= s->nx || y < 0 || y >= s->ny)
    return set_error(s, LBM_ERR_INVALID_ARG, "cell outside the grid");
  void* dst = s->box.out;
  if (!s->direct) {
    if (int rc = ensure_stage(s, kQ * 8)) return rc;
    dst = s->stage;
  }
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = probe_t<float>(s, x, y, dst); break;
    case LBM_FP64: rc = probe_t<double>(s, x, y, dst); break;
    case LBM_FP16_STORE: rc = probe_t<__half>(s, x, y, dst); break;
    case LBM_BF16_STORE: rc = probe_t<__nv_bfloat16>(s, x, y, dst); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  if (s->direct) {
    LBM_CUDA(s, cudaStreamSynchronize(s->stream));
    std::memcpy(out9, s->box.out, kQ * s->host_elem);
    return LBM_OK;
  }
  LBM_CUDA(s, cudaMemcpyAsync(out9, s->stage, kQ * s->host_elem, cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  return LBM_OK;
}

int lbm_set_body(lbm_solver* s, const uint8_t* body) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  if (!body) {
    cudaFree(s->body_d);
    s->body_d = nullptr;
    return LBM_OK;
  }
  const size_t n = static_cast<size_t>(s->nx) * s->ny;
  for (size_t c = 0; c < n; ++c)
    if (body[c] && !s->solid[c]) return set_error(s, LBM_ERR_INVALID_ARG, "body cells must be solid");
  // The box of the body's cells and their neighbours: first cell (periodic) and extent.
  int lo[2] = {s->nx, s->ny}, hi[2] = {-1, -1};
  for (int y = 0; y < s->ny; ++y)
    for (int x = 0; x < s->nx; ++x)
      if (body[static_cast<size_t>(y) * s->nx + x]) {
        lo[0] = std::min(lo[0], x), hi[0] = std::max(hi[0], x);
        lo[1] = std::min(lo[1], y), hi[1] = std::max(hi[1], y);
      }
  for (int d = 0; d < 2; ++d) {
    const int size = d == 0 ? s->nx : s->ny, extent = hi[d] < 0 ? 0 : hi[d] - lo[d] + 3;
    s->body_box[d] = extent >= size || extent == 0 ? 0 : lo[d] - 1;
    s->body_box[2 + d] = std::min(extent, size);
  }
  std::vector<uint32_t> words;
  pack_mask(body, s->nx, s->ny, s->g.mask_words, words);
  const size_t bytes = words.size() * sizeof(uint32_t);
  if (!s->body_d) LBM_CUDA(s, cudaMalloc(&s->body_d, bytes));
  LBM_CUDA(s, cudaMemcpyAsync(s->body_d, words.data(), bytes, cudaMemcpyHostToDevice, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  return LBM_OK;
}

int lbm_body_force(lbm_solver* s, double* fx, double* fy) {
  if (check(s) || !fx || !fy) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  if (!s->force_red) LBM_CUDA(s, cudaMalloc(&s->force_red, (2 * s->red_blocks + 2) * sizeof(double)));
  double* out = s->direct ? s->box.out : s->force_red + 2 * s->red_blocks;
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = body_force_t<float>(s, out); break;
    case LBM_FP64: rc = body_force_t<double>(s, out); break;
    case LBM_FP16_STORE: rc = body_force_t<__half>(s, out); break;
    case LBM_BF16_STORE: rc = body_force_t<__nv_bfloat16>(s, out); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  double f[2];
  if (!s->direct) LBM_CUDA(s, cudaMemcpyAsync(f, out, sizeof(f), cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  if (s->direct) std::memcpy(f, s->box.out, sizeof(f));
  *fx = f[0];
  *fy = f[1];
  return LBM_OK;
}

int lbm_check_finite(lbm_solver* s, int* finite) {
  if (check(s) || !finite) return set_error(s, LBM_ERR_INVALID_ARG, "null output");
  int* flag = s->direct ? const_cast<int*>(&s->box.bad) : reinterpret_cast<int*>(s->red + s->red_blocks + 2);
  if (s->direct)
    s->box.bad = 0;
  else
    LBM_CUDA(s, cudaMemsetAsync(flag, 0, sizeof(int), s->stream));
  int rc;
  switch (s->precision) {
    case LBM_FP32: rc = finite_t<float>(s, flag); break;
    case LBM_FP64: rc = finite_t<double>(s, flag); break;
    case LBM_FP16_STORE: rc = finite_t<__half>(s, flag); break;
    case LBM_BF16_STORE: rc = finite_t<__nv_bfloat16>(s, flag); break;
    default: rc = LBM_ERR_INVALID_ARG;
  }
  if (rc) return rc;
  int bad = 0;
  if (!s->direct) LBM_CUDA(s, cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  LBM_CUDA(s, cudaStreamSynchronize(s->stream));
  if (s->direct) bad = s->box.bad;
  *finite = bad ? 0 : 1;
  return LBM_OK;
}

int lbm_device_info(lbm_solver* s, char* buf, size_t size) {
  if (check(s) || !buf || size == 0) return set_error(s, LBM_ERR_INVALID_ARG, "null buffer");
  cudaDeviceProp prop{};
  int driver = 0, runtime = 0;
  LBM_CUDA(s, cudaGetDeviceProperties(&prop, s->device));
  LBM_CUDA(s, cudaDriverGetVersion(&driver));
  LBM_CUDA(s, cudaRuntimeGetVersion(&runtime));
  auto ver = [](int v) { return std::to_string(v / 1000) + "." + std::to_string((v % 1000) / 10); };
  static const char* names[] = {"fp32", "fp64", "fp16_store", "bf16_store"};
  const std::string info =
      "\"gpu\": \"" + std::string(prop.name) + "\", \"gpu_driver_cuda\": \"" + ver(driver) +
      "\", \"cuda_runtime\": \"" + ver(runtime) + "\", \"cuda_compiled\": \"" +
      ver(CUDART_VERSION) + "\", \"ecc\": " + std::to_string(prop.ECCEnabled) +
      ", \"sm_count\": " + std::to_string(s->sm_count) + ", \"block\": \"" +
      std::to_string(s->last_block ? s->last_block : s->block) + "x1\", \"grid\": " + std::to_string(s->last_grid) +
      ", \"variant\": \"b200_pull_vec" + std::to_string(s->vec) +
      "_v" + std::to_string(s->last_variant) + (s->variant < 0 ? "_auto" : "") + "\", \"precision\": \"" +
      names[s->precision] + "\"";
  std::snprintf(buf, size, "%s", info.c_str());
  return LBM_OK;
}

int lbm_get_shape(const lbm_solver* s, int* nx, int* ny, int* precision) {
  if (!s) return LBM_ERR_INVALID_ARG;
  if (nx) *nx = s->nx;
  if (ny) *ny = s->ny;
  if (precision) *precision = s->precision;
  return LBM_OK;
}

int lbm_set_launch(lbm_solver* s, int block_threads, int grid_blocks) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  const bool given = block_threads > 0;
  if (!given) block_threads = kStepThreads;
  if (block_threads % 32 != 0 || block_threads > kStepThreads || grid_blocks < 0)
    return set_error(s, LBM_ERR_INVALID_ARG, "block must be a multiple of 32 and <= 256");
  s->block = block_threads;
  s->block_set = given;
  s->grid = grid_blocks;
  lbm_b200::drop_step_graph(s);
  return LBM_OK;
}

int lbm_set_variant(lbm_solver* s, int variant) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  // 23 to 28 are of one storage form each; resident launches need a grid that fits.
  bool ok = variant >= -1 && variant <= kVariantF32Largest;
  if (variant == kVariantF32Large || variant == kVariantF32Largest) ok = s->elem == 4;
  if (variant == kVariantResident) ok = s->res.tx > 0;
  if (variant == kVariantF64Ring || variant == kVariantF64Direct) ok = s->elem == 8;
  if (variant == kVariant16Large) ok = s->elem == 2;
  if (!ok)
    return set_error(s, LBM_ERR_INVALID_ARG, "variant must be in [-1, 22], or a larger one of the solver's precision and grid");
  s->variant = variant;
  lbm_b200::drop_step_graph(s);
  return LBM_OK;
}

int lbm_state_view(lbm_solver* s, void** current, long long* plane_stride, int* row_pitch) {
  if (check(s)) return LBM_ERR_INVALID_ARG;
  if (current) *current = s->buf[s->cur];
  if (plane_stride) *plane_stride = s->g.plane;
  if (row_pitch) *row_pitch = s->g.pitch;
  return LBM_OK;
}

int lbm_test_set_consumer_wait_limit(unsigned polls) {
  const unsigned v = polls == 0 || polls >= lbm_b200::kSpinLimit ? lbm_b200::kSpinLimit : polls;
  lbm_b200::g_resident_polls = std::min(v, lbm_b200::kResidentPolls);
  const cudaError_t e = cudaMemcpyToSymbol(lbm_b200::c_consumer_wait_limit, &v, sizeof v);
  return e == cudaSuccess ? LBM_OK : LBM_ERR_CUDA;
}

}  // extern "C"
