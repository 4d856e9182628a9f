// Two x-adjacent FP32 cells per thread.
//
// A thread owns cells x0, x0 + 1 (x0 even) of one row: one 8-byte word per
// population. For c_x = 0 its inputs are one aligned word of the source row;
// for c_x = +-1 they are one value of that word and one more value at the row's
// periodic neighbour. Against one cell per thread that is three quarters of the
// loads, half of the stores and half of the address arithmetic per cell, and
// twice the bytes in flight per warp. A block covers kThreads consecutive words
// of one plane in memory order, so rows of any even length fill it. Direct loads
// of the shifted value beat taking it from the neighbouring lane by a shuffle
// (which also ties a warp to one row).
#pragma once

#include <cstdint>

#include "common.cuh"
#include "lattices.cuh"

namespace lbcube {

constexpr int kPairCells = 2;

// Blocks over the words of a plane: grid.x blocks of kThreads, grid.y planes
// from z0.
struct PairGrid {
  int nx, ny, nz;
  int pairs;       // words per row, nx / 2
  FastDiv by_row;  // in-plane word index -> row
  long long plane;
  int tiles;  // one-cell blocks per plane: a block covers kPairCells of them
  int z0;
};

inline PairGrid make_pair_grid(const Grid& g, int z0 = 0) {
  return PairGrid{g.nx, g.ny, g.nz, g.nx / 2, FastDiv((unsigned)(g.nx / 2)), g.plane, g.tiles, z0};
}

inline dim3 pair_grid_dims(const PairGrid& p, int planes) {
  return dim3((unsigned)((p.pairs * p.ny + kThreads - 1) / kThreads), (unsigned)planes);
}

// Rows of whole words in word-aligned buffers (an even plane keeps every
// population plane aligned), and a box that the rule takes. REDUCES: the kernel
// ends in a sum over the block.
template <bool REDUCES, class... P>
inline bool pairs_eligible(const Grid& g, const CellRule& rule, const P*... p) {
  return g.nx % 2 == 0 && ((((uintptr_t)p % 8) == 0) && ...) &&
         several_cells_pay(g.nx, g.ny, g.nz, kPairCells, REDUCES ? kThreads : 32, rule);
}

__device__ __forceinline__ bool pair_of(const PairGrid& g, int& x0, int& y, int& z) {
  const unsigned int c = blockIdx.x * (unsigned int)kThreads + threadIdx.x;
  y = (int)g.by_row(c);
  x0 = 2 * ((int)c - y * g.pairs);
  z = g.z0 + (int)blockIdx.y;
  return c < (unsigned int)(g.pairs * g.ny);
}

// The rows and wrapped neighbours of a pair.
struct PairRows {
  int x0, xl, xr;  // first cell, the row's periodic left and right neighbours of the pair
  int y[3], z[3];  // source row and plane for c = +1, 0, -1
  __device__ __forceinline__ PairRows(const PairGrid& g, int x, int yy, int zz) {
    x0 = x;
    xl = x == 0 ? g.nx - 1 : x - 1;
    xr = x + 2 == g.nx ? 0 : x + 2;
    y[0] = yy == 0 ? g.ny - 1 : yy - 1;
    y[1] = yy;
    y[2] = yy == g.ny - 1 ? 0 : yy + 1;
    z[0] = zz == 0 ? g.nz - 1 : zz - 1;
    z[1] = zz;
    z[2] = zz == g.nz - 1 ? 0 : zz + 1;
  }
  // In-plane offset of the row that population i is pulled from (< 2^31).
  template <class L, int i>
  __device__ __forceinline__ unsigned int row(const PairGrid& g) const {
    constexpr int ky = 1 - L::c[i][1], kz = 1 - L::c[i][2];
    return (unsigned int)((z[kz] * g.ny + y[ky]) * g.nx);
  }
};

// Pull-gather of all Q populations of the pair. FIRST: evict_first_loads.
template <class L, bool FIRST = false>
__device__ __forceinline__ void gather_pair(const float* __restrict__ cur, const PairGrid& g, const PairRows& r,
                                            float (&f)[2][L::Q]) {
  const size_t plane = (size_t)g.plane;
  const PullLoad<FIRST> load;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0];
    const float* row = cur + plane * i + r.template row<L, i>(g);
    const float2 w = load(reinterpret_cast<const float2*>(row + r.x0));
    if constexpr (cx == 0) {
      f[0][i] = w.x;
      f[1][i] = w.y;
    } else if constexpr (cx > 0) {  // source x - 1
      f[0][i] = load(row + r.xl);
      f[1][i] = w.x;
    } else {  // source x + 1
      f[0][i] = w.y;
      f[1][i] = load(row + r.xr);
    }
  });
}

// All Q populations of the pair itself.
template <class L>
__device__ __forceinline__ void load_pair(const float* __restrict__ cur, const PairGrid& g, int cell,
                                          float (&f)[2][L::Q]) {
  static_for<L::Q>([&](auto I) {
    const float2 w = __ldg(reinterpret_cast<const float2*>(cur + (size_t)g.plane * LB_I(I) + cell));
    f[0][LB_I(I)] = w.x;
    f[1][LB_I(I)] = w.y;
  });
}

template <int N>
__device__ __forceinline__ void store_pair(float* __restrict__ out, const PairGrid& g, int cell,
                                           const float (&f)[2][N]) {
  static_for<N>([&](auto I) {
    *reinterpret_cast<float2*>(out + (size_t)g.plane * LB_I(I) + cell) = make_float2(f[0][LB_I(I)], f[1][LB_I(I)]);
  });
}

// The adjoint of gather_pair: f[j][i] goes to the place the pair's cell j pulls
// population i from.
template <class L>
__device__ __forceinline__ void scatter_pair(float* __restrict__ out, const PairGrid& g, const PairRows& r,
                                             const float (&f)[2][L::Q]) {
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0];
    float* row = out + (size_t)g.plane * i + r.template row<L, i>(g);
    if constexpr (cx == 0) {
      *reinterpret_cast<float2*>(row + r.x0) = make_float2(f[0][i], f[1][i]);
    } else if constexpr (cx > 0) {
      row[r.xl] = f[0][i];
      row[r.x0] = f[1][i];
    } else {
      row[r.x0 + 1] = f[0][i];
      row[r.xr] = f[1][i];
    }
  });
}

// Pull-gather of the pair's 16-bit codes, one 32-bit word per population.
template <class L>
__device__ __forceinline__ void gather_code_pair(const unsigned short* __restrict__ cur, const PairGrid& g,
                                                 const PairRows& r, unsigned int (&w)[L::Q]) {
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0];
    const unsigned short* row = cur + (size_t)g.plane * i + r.template row<L, i>(g);
    const unsigned int own = __ldg(reinterpret_cast<const unsigned int*>(row + r.x0));
    if constexpr (cx == 0) w[i] = own;
    else if constexpr (cx > 0) w[i] = __byte_perm(__ldg(row + r.xl), own, 0x5410);
    else w[i] = __byte_perm(own, __ldg(row + r.xr), 0x5432);
  });
}

}  // namespace lbcube
