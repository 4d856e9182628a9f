// Pull collide-stream on shifted 16-bit populations, four x-adjacent cells per
// thread.
//
// A thread owns cells x0 .. x0 + 3 (x0 a multiple of 4) of one row, i.e. one
// 8-byte word of codes per population. For c_x = 0 its inputs are one aligned
// word of the source row; for c_x = +-1 they are that word and one more code at
// the row's periodic neighbour, joined by byte permutes. Every load is issued
// before the first value is used; the two cells of each 32-bit pair are then
// decoded, collided and encoded together (paired conversions; the stochastic
// rounding of a pair draws on both of its values, so pairs are always the cells
// (2k, 2k + 1) of a row).
//
// A block covers kThreads consecutive words of one plane in memory order, so
// rows of any length fill it; only x_extent a multiple of 4 and 8-byte aligned
// buffers are needed (the public contract of the 16-bit step).
//
// Bound by HBM bytes (76 B per D3Q19 cell) as long as the instructions of a
// cell leave room: a quarter of the memory instructions of one cell per thread,
// and few enough registers (kCodeBlocks resident blocks) that the warps of an SM
// keep about 90 KB of loads in flight. One step in us, against a kernel that
// staged whole rows in shared memory by bulk copies (and, where rows were no
// multiple of 8 cells, four cells per thread with shuffled neighbours, a warp
// per row): D3Q19 FP16 TRT 256^3 211.7 -> 193.1 (6.60 TB/s, a copy's rate),
// 128^3 32.1 -> 24.7, 64^3 15.6 -> 5.3; Q15 MRT 256^3 244 -> 207, 100 x 90 x 111
// 20.8 -> 12.9; E3M12 TRT 256^3 401 -> 282 (its integer codec). Two cells per
// thread: FP16 TRT 256^3 217.
#pragma once

#include <cstdint>

#include "codes.cuh"
#include "common.cuh"
#include "slab_faces.cuh"

namespace lbcube {

constexpr int kCodeCells = 4;  // cells per thread: one 8-byte word of codes

// Blocks over the words of a plane: grid.x = tiles, grid.y = planes from z0,
// z_step apart.
struct CodeGrid {
  int nx, ny, nz;
  int words;       // words per row, nx / 4
  FastDiv by_row;  // in-plane word index -> row
  long long plane;
  int z0, z_step;
};

inline CodeGrid make_code_grid(const Grid& g, int z0 = 0, int z_step = 1) {
  CodeGrid c;
  c.nx = g.nx;
  c.ny = g.ny;
  c.nz = g.nz;
  c.words = g.nx / kCodeCells;
  c.by_row = FastDiv((unsigned)c.words);
  c.plane = g.plane;
  c.z0 = z0;
  c.z_step = z_step;
  return c;
}

// When the coupled fluid + A + B -> C step on 16-bit codes takes four cells per
// thread, `resident` being how many blocks of its one-cell kernel an SM holds. The
// four-cell kernel is straight-line code for four collisions and reactions at 5
// resident blocks: 4.2 us for the smallest box, where one cell per thread takes 2.
// One step in us, one cell -> four, at one-cell blocks per SM: D3Q19 FP16 TRT 32^3
// (1.7) 2.6 -> 4.6, 48^3 (5.8) 5.7 -> 5.0, 64 x 64 x 32 (6.9) 5.7 -> 5.1, 56^3 (9.5) 6.4 ->
// 8.0, 64^3 (13.8) 8.4 -> 8.1, 80^3 (27) 15.4 -> 11.7; E3M12 64^3 12.2 -> 14.2, 76^3 (23.6)
// 20.0 -> 20.3, 80^3 22.9 -> 22.4; Q15 MRT 64^3 9.9 -> 10.6, 80^3 17.7 -> 16.6. D2Q9 FP16
// TRT 320^2 (5.4) 3.25 -> 3.37, 352^2 (6.5) 3.7 -> 3.4, 512^2 6.4 -> 5.7; E3M12 512^2 8.3 ->
// 9.2, 704^2 (26) 13.9 -> 12.5; Q15 640^2 (21.6) 9.4 -> 9.7, 704^2 11.1 -> 10.6.
template <class FL, int FMT>
inline CellRule coupled_codes_rule(int resident) {
  constexpr bool kFloats = FMT == kF16S || FMT == kBF16S;
  constexpr double from = FL::Q == 9 ? (kFloats ? 6 : 24) : (kFloats ? 13 : 26);
  constexpr double hi = kFloats ? 2.5 : 2;  // half of 5; the integer codecs lose the wave at 52^3 (2.1)
  return resident <= 0 ? CellRule{from} : CellRule{from, resident / 2.0 < 4 ? 4 : resident / 2.0, hi};
}

inline bool codes_eligible(const Grid& g, const void* a, const void* b) {
  return g.nx % kCodeCells == 0 && (uintptr_t)a % 8 == 0 && (uintptr_t)b % 8 == 0;
}

// The word, row and plane of this thread; false for the idle threads of a
// plane's last block.
__device__ __forceinline__ bool word_of(const CodeGrid& g, int& x0, int& y, int& z) {
  const unsigned int c = blockIdx.x * (unsigned int)blockDim.x + threadIdx.x;
  y = (int)g.by_row(c);
  x0 = kCodeCells * ((int)c - y * g.words);
  z = g.z0 + (int)blockIdx.y * g.z_step;
  return c < (unsigned int)(g.words * g.ny);
}

// The codes of cells x0 .. x0 + 3 pulled along c_x from `row`: two pairs.
template <int CX>
__device__ __forceinline__ void pull_codes(const unsigned short* __restrict__ row, int x0, int xl, int xr,
                                           unsigned int (&w)[2]) {
  const uint2 own = __ldg(reinterpret_cast<const uint2*>(row + x0));
  if constexpr (CX == 0) {
    w[0] = own.x;
    w[1] = own.y;
  } else if constexpr (CX > 0) {  // cells x0-1 .. x0+2
    const unsigned int left = __ldg(row + xl);
    w[0] = __byte_perm(left, own.x, 0x5410);
    w[1] = __byte_perm(own.x, own.y, 0x5432);
  } else {  // cells x0+1 .. x0+4
    const unsigned int right = __ldg(row + xr);
    w[0] = __byte_perm(own.x, own.y, 0x5432);
    w[1] = __byte_perm(own.y, right, 0x5432);
  }
}

// All Q populations of the thread's four cells. SLAB: a z-slab of a box; at
// plane 0 the c_z = +1 rows come from halo_lo, at plane nz - 1 the c_z = -1 rows
// from halo_hi, instead of the periodic wrap (SlabArgs).
template <class L, bool SLAB = false>
__device__ __forceinline__ void gather_words(const unsigned short* __restrict__ cur, const CodeGrid& g,
                                             int x0, int y, int z, unsigned int (&raw)[L::Q][2],
                                             const SlabArgs<unsigned short>& slab = {}) {
  const int xl = x0 == 0 ? g.nx - 1 : x0 - 1;
  const int xr = x0 + kCodeCells == g.nx ? 0 : x0 + kCodeCells;
  const int ym = y == 0 ? g.ny - 1 : y - 1, yp = y == g.ny - 1 ? 0 : y + 1;
  const int zm = z == 0 ? g.nz - 1 : z - 1, zp = z == g.nz - 1 ? 0 : z + 1;
  const size_t plane = (size_t)g.plane;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cx = L::c[i][0], cy = L::c[i][1], cz = L::c[i][2];
    const int sy = cy == 0 ? y : (cy > 0 ? ym : yp);
    const int sz = cz == 0 ? z : (cz > 0 ? zm : zp);
    const unsigned short* row = cur + plane * i + (unsigned int)((sz * g.ny + sy) * g.nx);
    if constexpr (SLAB && cz > 0) {
      if (z == 0) row = slab.halo_lo + (size_t)(zslot_of<L>(i) * g.ny + sy) * g.nx;
    } else if constexpr (SLAB && cz < 0) {
      if (z == g.nz - 1) row = slab.halo_hi + (size_t)(zslot_of<L>(i) * g.ny + sy) * g.nx;
    }
    pull_codes<cx>(row, x0, xl, xr, raw[i]);
  });
}

template <class L, class S, int CT, bool SLAB>
__device__ __forceinline__ void code_step_body(const unsigned short* __restrict__ cur,
                                               unsigned short* __restrict__ nxt, const CodeGrid& g,
                                               float omega, float omega_minus, const typename S::Params& p,
                                               const SlabArgs<unsigned short>& slab) {
  pdl_enter();
  int x0, y, z;
  if (!word_of(g, x0, y, z)) return;
  unsigned int raw[L::Q][2];
  gather_words<L, SLAB>(cur, g, x0, y, z, raw, slab);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float va[L::Q], vb[L::Q];
    static_for<L::Q>([&](auto I) {
      const float2 d = S::template decode_pair<L, LB_I(I)>(raw[LB_I(I)][h], p);
      va[LB_I(I)] = d.x;
      vb[LB_I(I)] = d.y;
    });
    S::template collide_cell<L, CT>(va, omega, omega_minus, p);
    S::template collide_cell<L, CT>(vb, omega, omega_minus, p);
    static_for<L::Q>([&](auto I) {
      raw[LB_I(I)][h] = S::template encode_pair<L, LB_I(I)>(va[LB_I(I)], vb[LB_I(I)], p);
    });
  }
  const size_t plane = (size_t)g.plane;
  const int cell = (z * g.ny + y) * g.nx + x0;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int cz = L::c[i][2];
    const uint2 w = make_uint2(raw[i][0], raw[i][1]);
    *reinterpret_cast<uint2*>(nxt + plane * i + cell) = w;
    // the populations leaving through a face, at the cells' own (x, y)
    if constexpr (SLAB && cz > 0) {
      if (z == g.nz - 1)
        *reinterpret_cast<uint2*>(slab.send_hi + (size_t)(zslot_of<L>(i) * g.ny + y) * g.nx + x0) = w;
    } else if constexpr (SLAB && cz < 0) {
      if (z == 0) *reinterpret_cast<uint2*>(slab.send_lo + (size_t)(zslot_of<L>(i) * g.ny + y) * g.nx + x0) = w;
    }
  });
}

// Resident blocks of kThreads per SM that the register allocation must allow.
// D3Q19 on the deviations: 6 (80 registers; FP16 TRT 256^3, 20 steps with encode
// and decode, 4.63 ms against 4.74 at 5, 5.02 at 7 and 6.08 at 8, which spill).
// Decoded D3Q19 (RLBM): 5 (64 x 94 x 59, 9 steps: 134 us against 147 at 6).
// D3Q27: 4 (MRT, 312 x 244 x 151, 6 steps: 5.19 ms against 5.35 at 3, 5.45 at 5).
// D2Q9: 8 (level from 6 to 12).
template <class L, class S>
constexpr int kCodeBlocks = L::Q == 9 ? 8 : L::Q == 27 ? 4 : S::kDecoded ? 5 : 6;

template <class L, class S, int CT>
__global__ void __launch_bounds__(kThreads, kCodeBlocks<L, S>)
    code_step_kernel(const unsigned short* __restrict__ cur, unsigned short* __restrict__ nxt, CodeGrid g,
                     float omega, float omega_minus, typename S::Params p) {
  code_step_body<L, S, CT, false>(cur, nxt, g, omega, omega_minus, p, {});
}

// The face planes of a z-slab.
template <class L, class S, int CT>
__global__ void __launch_bounds__(kThreads)
    code_step_slab_kernel(const unsigned short* __restrict__ cur, unsigned short* __restrict__ nxt,
                          CodeGrid g, float omega, float omega_minus, typename S::Params p,
                          SlabArgs<unsigned short> slab) {
  code_step_body<L, S, CT, true>(cur, nxt, g, omega, omega_minus, p, slab);
}

// `planes` planes from z0, z_step apart; slab: their SLAB form.
template <class L, class S, int CT>
inline cudaError_t launch_code_step(const Grid& g, cudaStream_t stream, const unsigned short* cur,
                                    unsigned short* nxt, float omega, float omega_minus,
                                    const typename S::Params& p, int z0, int planes, int z_step = 1,
                                    const SlabArgs<unsigned short>* slab = nullptr) {
  const CodeGrid cg = make_code_grid(g, z0, z_step);
  const unsigned words = (unsigned)(cg.words * g.ny);
  const dim3 grid((words + kThreads - 1) / kThreads, (unsigned)planes), block(kThreads);
  if (slab != nullptr)
    return launch_pdl(code_step_slab_kernel<L, S, CT>, grid, block, 0, stream, cur, nxt, cg, omega,
                      omega_minus, p, *slab);
  return launch_pdl(code_step_kernel<L, S, CT>, grid, block, 0, stream, cur, nxt, cg, omega, omega_minus, p);
}

}  // namespace lbcube
