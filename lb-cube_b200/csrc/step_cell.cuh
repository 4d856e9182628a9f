// Fused pull-scheme collide-stream step for D2Q9 / D3Q19 / D3Q27 fluids: one
// cell per thread, and two FP32 cells per thread (pairs.cuh); shared by the
// periodic step (fluid_step.cu) and the interior planes of the slab step
// (slab.cu).
//
// Replaces kernel_step (src/lattice_cuda.cu:149-213). In the one-cell form a
// thread owns one destination cell: it gathers the Q incoming populations
// f_i(x - c_i) from the current buffer (periodic wrap by compare-and-select on
// 32-bit coordinates instead of the reference's 64-bit modulo), collides in
// registers and writes the Q results to the next buffer at its own cell. A warp
// covers 32 consecutive cells, so each of the Q gathers and Q stores is one
// coalesced segment (shifted by at most one element for c_x != 0, which the
// L1/L2 sector reuse absorbs). Planes g.z0 + k * g.zs (k < gridDim.y) are stepped.
#pragma once
#include "collide.cuh"
#include "common.cuh"
#include "diag.cuh"
#include "packed.cuh"
#include "pairs.cuh"

namespace lbcube {

// FIRST: evict_first_loads.
template <class L, class Real, int CT, bool FIRST>
__device__ __forceinline__ void step_cell(const Real* __restrict__ cur, Real* __restrict__ nxt,
                                          const Grid& g, int x, int y, int z, Real omega,
                                          Real omega_minus, Real (&f)[L::Q]) {
  const int xm = x == 0 ? g.nx - 1 : x - 1, xp = x == g.nx - 1 ? 0 : x + 1;
  const int ym = y == 0 ? g.ny - 1 : y - 1, yp = y == g.ny - 1 ? 0 : y + 1;
  const int zm = z == 0 ? g.nz - 1 : z - 1, zp = z == g.nz - 1 ? 0 : z + 1;
  const size_t plane = (size_t)g.plane;
  const PullLoad<FIRST> load;

  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0], cy = L::c[i][1], cz = L::c[i][2];
    // pull: source = destination - c_i (lattice_core.hpp:70-78)
    const int sx = cx == 0 ? x : (cx > 0 ? xm : xp);
    const int sy = cy == 0 ? y : (cy > 0 ? ym : yp);
    const int sz = cz == 0 ? z : (cz > 0 ? zm : zp);
    f[i] = load(cur + plane * i + ((sz * g.ny + sy) * g.nx + sx));
  });

  collide<L, Real, CT>(f, omega, omega_minus);

  const int cell = (z * g.ny + y) * g.nx + x;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    nxt[plane * i + cell] = f[i];
  });
}

// DIAG: also reduce the diagnostics of the written state over the block
// (diag.cuh): in the pull scheme the populations a thread writes are exactly the
// next buffer's populations of its own cell, so this costs no memory traffic.
template <class L, class Real, int CT, bool DIAG, bool FIRST>
__global__ void __launch_bounds__(kThreads)
    fluid_step_kernel(const Real* __restrict__ cur, Real* __restrict__ nxt, Grid g, Real omega,
                      Real omega_minus, double* __restrict__ partials) {
  pdl_enter();
  int x, y, z;
  const bool active = cell_of(g, x, y, z);
  Real f[L::Q];
  if constexpr (DIAG) {
    DiagAcc acc;
    if (active) {
      step_cell<L, Real, CT, FIRST>(cur, nxt, g, x, y, z, omega, omega_minus, f);
      diag_cell<L>(f, acc);
    }
    diag_block_to(acc, partials + block_linear() * kDiagPartials);
  } else {
    if (!active) return;
    step_cell<L, Real, CT, FIRST>(cur, nxt, g, x, y, z, omega, omega_minus, f);
  }
}

// The Q population planes of a buffer as separate base pointers, passed as
// kernel parameters (read from the constant bank): every gather and store is
// then one wide multiply-add of a 32-bit in-plane offset, where base + plane * i
// otherwise costs 64-bit arithmetic per population. Used for MRT on D3Q19 and
// D3Q27, where it measured faster (A/B, same box, bit-identical outputs:
// D3Q19 FP64 MRT 0.94 -> 0.98 of the copy bandwidth at 256^3, D3Q27 FP32 MRT
// 0.56 -> 0.585 at 224^3; D3Q19 FP32 MRT and D3Q27 BGK level; RLBM 1.5-7 % and
// D2Q9 MRT 2.5 % slower, so those keep fluid_step_kernel).
template <class L, class Real, int CT>
constexpr bool kUsePlanes = CT == kMRT && L::Q >= 19;
template <class Real, int Q>
struct Planes {
  Real* p[Q];
};
template <class Real, int Q>
inline Planes<Real, Q> planes_of(Real* base, const Grid& g) {
  Planes<Real, Q> r;
  for (int i = 0; i < Q; ++i) r.p[i] = base + (size_t)g.plane * i;
  return r;
}

// fluid_step_kernel (no diagnostics) on plane pointers: the same gather,
// collision and stores, so the same bits.
template <class L, class Real, int CT, bool FIRST>
__global__ void __launch_bounds__(kThreads)
    fluid_step_planes_kernel(const Planes<const Real, L::Q> cur, const Planes<Real, L::Q> nxt,
                             Grid g, Real omega, Real omega_minus) {
  pdl_enter();
  int x, y, z;
  if (!cell_of(g, x, y, z)) return;
  const int xm = x == 0 ? g.nx - 1 : x - 1, xp = x == g.nx - 1 ? 0 : x + 1;
  const int ym = y == 0 ? g.ny - 1 : y - 1, yp = y == g.ny - 1 ? 0 : y + 1;
  const int zm = z == 0 ? g.nz - 1 : z - 1, zp = z == g.nz - 1 ? 0 : z + 1;
  Real f[L::Q];
  const PullLoad<FIRST> load;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0], cy = L::c[i][1], cz = L::c[i][2];
    const int sx = cx == 0 ? x : (cx > 0 ? xm : xp);
    const int sy = cy == 0 ? y : (cy > 0 ? ym : yp);
    const int sz = cz == 0 ? z : (cz > 0 ? zm : zp);
    f[i] = load(cur.p[i] + ((sz * g.ny + sy) * g.nx + sx));
  });
  collide<L, Real, CT>(f, omega, omega_minus);
  const int cell = (z * g.ny + y) * g.nx + x;
  static_for<L::Q>([&](auto I) { nxt.p[LB_I(I)][cell] = f[LB_I(I)]; });
}

// ---- two FP32 cells per thread ---------------------------------------------------
// One step in us, one cell per thread -> two: D3Q19 TRT 256^3 394 -> 380 (6.7 TB/s,
// a copy's rate), 160^3 100 -> 97, 96^3 22.1 -> 20.4; MRT 128^3 59 -> 55; RLBM
// 128^3 69 -> 60; D3Q27 BGK 128^3 74 -> 72, RLBM 105 -> 95; D2Q9 BGK 1448^2 24.7 ->
// 20.5. Against the kernel that exchanged x-neighbours by shuffles, a warp per
// row: D3Q19 TRT 256^3 383, 160^3 118, 96^3 29.7. Four cells per thread: level
// at 256^3, slower below.
//
// Resident blocks of kThreads per SM that the register allocation must allow
// (0: the compiler's choice): D3Q19 7 (72 registers; TRT 180 x 170 x 190 140 us
// against 143 at 6 and 142 at 8; MRT 151, 159 and 154), RLBM, D2Q9 and D3Q27 the
// compiler's (D3Q27 BGK 72 x 70 x 68 9.8 us against 11.0 at 4).
// D3Q27 MRT, in packed arithmetic, 4 (128 registers; 128^3 in a loop of its own
// 83.6 us against 92 at 3 and 86 at 5, which spills).
template <class L, int CT>
constexpr int kPairBlocks = L::Q == 27 && CT == kMRT ? 4 : L::Q == 19 && CT != kRLBM ? 7 : 0;
// From how many one-cell blocks per SM on: what the SMs hold at once. D3Q19 12:
// MRT 56^3 (9.5 blocks per SM) 6.1 -> 6.5 us, 64^3 (13.8) 7.3 -> 6.6. D2Q9 16: MRT
// 512^2 (13.8) 4.2 -> 5.2, 600^2 (19) 5.1 -> 5.0, 724^2 6.5 -> 5.8. D3Q27 likewise:
// BGK 64^3 (13.8) level, 72^3 (19.9) 11.5 -> 10.4; its RLBM later: 72^3 18.0 -> 18.4,
// 88^3 (36) 36.6 -> 33.7; and its MRT: 60 x 62 x 64 (13.4) 11.9 -> 12.4, 72^3 17.7 ->
// 18.0, 88 x 90 x 86 (35) 30.8 -> 29.4. Between, D3Q19 BGK, TRT and MRT: from 6 (half of
// the 12 resident one-cell blocks) while the pairs' blocks stay within half of their
// 7: 64 x 64 x 32 (6.9) BGK 4.8 -> 3.8, TRT 5.2 -> 4.0, MRT 5.3 -> 4.5; BGK and TRT up to
// half of 8, on a kernel of that budget (64 registers, 6 % slower where both fit):
// 64 x 64 x 36 BGK 4.95 -> 4.1, 52^3 TRT 5.3 -> 4.2.
constexpr int kWindowBlocks = 8;
template <class L, int CT>
constexpr CellRule kPairRule = L::Q != 19 ? CellRule{L::Q == 27 && (CT == kRLBM || CT == kMRT) ? 30.0 : 16.0}
                               : CT == kRLBM ? CellRule{12}
                                             : CellRule{12, 6, CT == kMRT ? 3.5 : kWindowBlocks / 2.0};
// The diagnostics form of the D3Q27 step keeps one cell per thread: its FP64 sums
// cost a pair more registers than the saved loads are worth (96^3: TRT 41.7 us
// against 43.2, MRT 54.6 against 56.9, RLBM 56.2 against 57.9).
template <class L, class Real, bool DIAG>
constexpr bool kUsePairs = sizeof(Real) == 4 && !(DIAG && L::Q == 27);

template <class L, int CT, bool DIAG, bool FIRST, int BLOCKS>
__global__ void __launch_bounds__(kThreads, BLOCKS)
    fluid_step_pair_kernel(const float* __restrict__ cur, float* __restrict__ nxt, PairGrid g, float omega,
                           float omega_minus, double* __restrict__ partials) {
  pdl_enter();
  int x0, y, z;
  const bool active = pair_of(g, x0, y, z);
  DiagAcc acc;
  if (active) {
    float f[2][L::Q];
    gather_pair<L, FIRST>(cur, g, PairRows(g, x0, y, z), f);
    collide_pair<L, CT>(f, omega, omega_minus);
    store_pair(nxt, g, (z * g.ny + y) * g.nx + x0, f);
    if constexpr (DIAG) {
#pragma unroll
      for (int j = 0; j < 2; ++j) diag_cell<L>(f[j], acc);
    }
  }
  if constexpr (DIAG)
    diag_block_to(acc, partials + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * kDiagPartials);
}

// The blocks of the one-cell step. D2Q9 FP64 BGK (48 registers), where the populations
// stay in L2 and the launch is past half of the resident blocks: blocks of 96, of
// which an SM holds 14 (42 warps) where it holds 10 of 128 (40), and which rows of 96
// and 544 cells fill. 544 x 768 (22 blocks per SM) 6.67 -> 6.48 us, 96 x 4096 6.34 -> 6.07,
// 512^2 4.68 -> 4.46, 384^2 (7.8) 3.59 -> 3.50; 320^2 (5.4) 3.37 -> 3.41, 800 x 900 (38)
// 11.9 -> 12.0, 2048^2 91.4 -> 92.4. TRT and MRT level at 544 x 768, 3 % slower at 512^2.
template <class L, class Real, int CT>
inline Grid step_grid(const Grid& g) {
  if (sizeof(Real) == 8 && L::Q == 9 && CT == kBGK && g.launched() > 7LL * kSMs && g.launched() <= 30LL * kSMs) {
    Grid c = g;
    c.bx = 96;
    c.tiles = (int)(((long long)g.nx * g.ny + c.bx - 1) / c.bx);
    return c;
  }
  return latency_grid<L, Real>(g, kStepSpread);
}

// One step of planes g.z0 .. g.z0 + planes - 1 on the kernel that is the faster one
// for this lattice, operator, precision and row length. DIAG: with the
// diagnostics' partials, whose count goes to *count (over every plane; at most
// g.launched()).
template <class L, class Real, int CT, bool DIAG, bool FIRST>
inline cudaError_t launch_step(const Grid& g, int planes, const Real* cur, Real* nxt, Real omega,
                               Real omega_minus, double* partials, long long* count, cudaStream_t s) {
  // programmatic dependent launches (the kernels open with pdl_enter)
  if constexpr (kUsePairs<L, Real, DIAG>) {
    // the range below `from` is that of a loop of this launch alone: with a slab's face
    // launch after it one cell per thread is faster (64 x 64 x 32 MRT 6.5 us, pairs 7.0)
    constexpr CellRule rule = kPairRule<L, CT>;
    if (pairs_eligible<DIAG>(g, planes == g.nz ? rule : CellRule{rule.from}, cur, nxt)) {
      const PairGrid pg = make_pair_grid(g, g.z0);
      const dim3 grid = pair_grid_dims(pg, planes);
      if constexpr (DIAG) *count = (long long)grid.x * planes;
      auto run = [&](auto blocks) {
        return launch_pdl(fluid_step_pair_kernel<L, CT, DIAG, FIRST, decltype(blocks)::value>, grid, dim3(kThreads), 0,
                          s, cur, nxt, pg, omega, omega_minus, partials);
      };
      if constexpr (kPairRule<L, CT>.hi == kWindowBlocks / 2.0 && !FIRST) {
        const bool window = g.launched() <= (long long)kPairRule<L, CT>.from * kSMs;
        if (window && 2LL * grid.x * planes > (long long)kPairBlocks<L, CT> * kSMs)
          return run(std::integral_constant<int, kWindowBlocks>{});
      }
      return run(std::integral_constant<int, kPairBlocks<L, CT>>{});
    }
  }
  const Grid gl = DIAG || planes != g.nz ? g : step_grid<L, Real, CT>(g);
  const dim3 grid((unsigned)gl.tiles, (unsigned)planes), block(block_dims(gl));
  if constexpr (DIAG) *count = (long long)g.tiles * planes;
  if constexpr (kUsePlanes<L, Real, CT> && !DIAG)
    return launch_pdl(fluid_step_planes_kernel<L, Real, CT, FIRST>, grid, block, 0, s,
                      planes_of<const Real, L::Q>(cur, gl), planes_of<Real, L::Q>(nxt, gl), gl, omega,
                      omega_minus);
  else
    return launch_pdl(fluid_step_kernel<L, Real, CT, DIAG, FIRST>, grid, block, 0, s, cur, nxt, gl, omega,
                      omega_minus, partials);
}

}  // namespace lbcube
