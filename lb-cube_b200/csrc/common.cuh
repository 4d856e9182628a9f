// Launch geometry and argument validation shared by every kernel family.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "lattices.cuh"

namespace lbcube {

// Most threads per block. In the one-cell-per-thread kernels a block covers
// kThreads consecutive cells of one z plane.
constexpr int kThreads = 128;
constexpr int kSMs = 148;

// Division of n < 2^31 by an invariant d < 2^31 as one high product and a
// shift: mul = ceil(2^(31 + l) / d) with l = ceil(log2 d), so that mul < 2^32 and
// mul d - 2^(31 + l) < 2^l, which makes floor(n mul / 2^(31 + l)) the quotient for
// every n < 2^31 (T. Granlund, P. L. Montgomery, "Division by Invariant
// Integers using Multiplication", PLDI 1994).
struct FastDiv {
  unsigned int mul = 0, shift = 0;
  FastDiv() = default;
  explicit FastDiv(unsigned int d) {
    while ((1ull << shift) < d) ++shift;
    mul = (unsigned int)(((1ull << (31 + shift)) + d - 1) / d);
  }
  __host__ __device__ __forceinline__ unsigned int operator()(unsigned int n) const {
#ifdef __CUDA_ARCH__
    return __umulhi(2u * n, mul) >> shift;
#else
    return (unsigned int)(((unsigned long long)(2u * n) * mul) >> 32) >> shift;
#endif
  }
};

// Domain extents and the block decomposition: grid.x = tiles blocks of bx
// threads over the nx * ny cells of a plane in memory order, grid.y = nz. Rows
// share blocks, so only the last block of a plane has idle threads: rows of
// 201 cells cost 201 lanes, where blocks of whole rows took 256 (2 x 128), and
// rows of 135 took 192. Against such blocks: D3Q19 FP32 MRT on 201 x 130 x 75
// 63.4 -> 56.6 us per step, TRT step + scalar step on 135 x 128 x 90 86.4 ->
// 74.1 us, rows of a multiple of 128 level.
struct Grid {
  int nx, ny, nz;
  int tiles;        // blocks per plane
  int bx;           // threads per block
  FastDiv by_nx;    // in-plane cell index -> row
  long long plane;  // cells per population plane, nx * ny * nz (< 2^31)
  long long row_blocks;  // ceil(nx / kThreads) * ny * nz: the partials contract below
  int z0 = 0;       // first z plane of the launch
  int zs = 1;       // planes between consecutive blockIdx.y: z = z0 + blockIdx.y * zs (both face
                    // planes of a slab in one launch: z0 = 0, zs = nz - 1)

  // Partial sums that a caller's scratch buffer must hold (the public sizes:
  // one per 128-cell segment of a row), and how many of them a launch over
  // every plane writes: launched() <= blocks().
  __host__ __device__ long long blocks() const { return row_blocks; }
  __host__ __device__ long long launched() const { return (long long)tiles * nz; }
};

// The z plane of this block.
__device__ __forceinline__ int plane_of(const Grid& g) { return g.z0 + (int)blockIdx.y * g.zs; }

__device__ __forceinline__ bool cell_of(const Grid& g, int& x, int& y, int& z) {
  const unsigned int c = blockIdx.x * (unsigned int)g.bx + threadIdx.x;
  y = (int)g.by_nx(c);
  x = (int)c - y * g.nx;
  z = plane_of(g);
  return c < (unsigned int)(g.nx * g.ny);
}

// Linear block index used to address per-block partial sums.
__device__ __forceinline__ long long block_linear() {
  return (long long)blockIdx.y * gridDim.x + blockIdx.x;
}

// The load of a pulled population, through the read-only path; FIRST: with the
// L2 policy that evicts its line first.
template <bool FIRST>
struct PullLoad {
  unsigned long long policy = 0;
  __device__ __forceinline__ PullLoad() {
    if constexpr (FIRST) asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  }
  template <class T>
  __device__ __forceinline__ T operator()(const T* p) const {
    if constexpr (!FIRST) {
      return __ldg(p);
    } else if constexpr (std::is_same_v<T, float>) {
      float v;
      asm volatile("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
      return v;
    } else if constexpr (std::is_same_v<T, float2>) {
      float2 v;
      asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;"
                   : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(policy));
      return v;
    } else {
      static_assert(std::is_same_v<T, double>, "float, float2 or double");
      double v;
      asm volatile("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy));
      return v;
    }
  }
};

// Programmatic dependent launch. pdl_enter() at the top of a kernel waits
// until the grid it depends on has completed and its writes are visible (a
// no-op unless the kernel was launched with the programmatic-serialization
// attribute), then lets the next launch in the stream be scheduled, so that
// launch's blocks take the SMs that this grid's last blocks free instead of
// waiting for the whole grid to drain. launch_pdl launches with that attribute.
#ifndef LBCUBE_PDL
#define LBCUBE_PDL 1
#endif
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t s, Args&&... args) {
  if (!LBCUBE_PDL) {
    kernel<<<grid, block, smem, s>>>(std::forward<Args>(args)...);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// When a launch of several adjacent cells per thread beats one cell per thread. In
// `blocks per SM` of kThreads-thread blocks: `one` of the one-cell launch, `many` of
// the other.
// * from: above this many one-cell blocks per SM, about what the SMs hold at once or
//   more; below it the one-cell launch's many threads hide more latency than the
//   saved instructions are worth.
// * lo, hi: also where one > lo and many <= hi. The next launch of a stream waits
//   on the SMs while one runs (pdl_enter), so a launch goes without a second wave
//   up to half of the resident blocks: between the halves of the two kernels
//   (lo, hi) only the one-cell launch takes the second wave.
// * unit: a plane's threads fill whole blocks (kThreads) where idle warps wait at a
//   barrier or hold a large block's registers, whole warps (32) elsewhere; a plane
//   that this pads by over 15 % more than the one-cell launch keeps one cell per thread.
struct CellRule {
  double from, lo = 0, hi = 0;
};
inline bool several_cells_pay(int nx, int ny, int nz, int cells, int unit, const CellRule& r) {
  const long long plane = (long long)nx * ny, threads = plane / cells;
  auto up = [](long long n, long long to) { return (n + to - 1) / to; };
  const double one = (double)up(plane, kThreads) * nz / kSMs, many = (double)up(threads, kThreads) * nz / kSMs;
  if (one > r.lo && many <= r.hi) return true;
  return one > r.from && 20 * up(threads, unit) * cells <= 23 * up(plane, unit);
}

// How many blocks of kThreads an SM holds of a kernel: a property of the compiled
// kernel, asked for until it is known (0: it cannot be told).
template <auto* kernel>
inline int resident_blocks() {
  static std::atomic<int> known{0};
  int n = known.load(std::memory_order_relaxed);
  if (n != 0) return n;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThreads, 0) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  known.store(n, std::memory_order_relaxed);
  return n;
}

inline dim3 grid_dims(const Grid& g) { return dim3((unsigned)g.tiles, (unsigned)g.nz, 1); }
inline unsigned block_dims(const Grid& g) { return (unsigned)g.bx; }

// Validation in the reference's order (src/lattice_cuda.cu:488-503), then the
// engine's own limits. On success fills `g`.
inline cudaError_t validate_domain(bool any_null, unsigned bx, unsigned by, unsigned bz, int dims,
                                   size_t nx, size_t ny, size_t nz, Grid& g) {
  if (any_null) return cudaErrorInvalidDevicePointer;
  if (bx == 0 || by == 0 || bz == 0) return cudaErrorInvalidConfiguration;
  if (dims == 2) nz = 1;
  if (nx == 0 || ny == 0 || nz == 0) return cudaErrorInvalidValue;
  if (nx > (size_t)INT_MAX || ny > (size_t)INT_MAX || nz > 65535) return cudaErrorInvalidValue;
  const unsigned long long cells = (unsigned long long)nx * ny;
  if (cells > (unsigned long long)INT_MAX || cells * nz > (unsigned long long)INT_MAX)
    return cudaErrorInvalidValue;
  g.nx = (int)nx;
  g.ny = (int)ny;
  g.nz = (int)nz;
  g.plane = (long long)(cells * nz);
  const long long segments = ((long long)nx + kThreads - 1) / kThreads * (long long)ny;
  if (segments > (long long)INT_MAX) return cudaErrorInvalidValue;
  g.row_blocks = segments * (long long)nz;
  g.bx = (int)(cells < kThreads ? (cells + 31) / 32 * 32 : kThreads);
  g.tiles = (int)((cells + g.bx - 1) / g.bx);
  g.by_nx = FastDiv((unsigned)nx);
  return cudaSuccess;
}

// A grid of fewer than `below` blocks per SM with smaller blocks, whole warps, until it
// has `upto` per SM, as far as the partials contract allows (launched() <= blocks()).
// A small box is bound by latency: more and smaller blocks reach more SMs, and a
// block's sums cross fewer warps; launches bound by neither lose to it (FP32 D3Q19
// BGK step 32^3 2.1 -> 2.5 us).
inline Grid spread(Grid g, double below, int upto) {
  const long long cells = (long long)g.nx * g.ny;
  auto launch_blocks = [&](int bx) { return (cells + bx - 1) / bx * g.nz; };
  if ((double)g.launched() >= below * kSMs) return g;
  while (g.bx > 32 && launch_blocks(g.bx) < (long long)upto * kSMs) {
    const int smaller = (g.bx / 2 + 31) / 32 * 32;
    if (launch_blocks(smaller) > g.row_blocks) break;
    g.bx = smaller;
  }
  g.tiles = (int)((cells + g.bx - 1) / g.bx);
  return g;
}

// The blocks of a statistics launch, whose partials the second pass counts from
// the extents alone. Coupled step with statistics, blocks of 128 -> these, us: D3Q19
// FP64 BGK 16^3 3.85 -> 3.25, 32^3 (1.7 blocks per SM) 4.70 -> 4.0, 40^3 (3.4) 7.0 -> 7.3
// and so left alone; FP32 TRT 16^3 3.4 -> 3.0.
inline Grid stats_grid(const Grid& g) { return spread(g, 2, 4); }

// The blocks of a 3-D FP64 launch over a whole box without partials, planes of less
// than a block apart (8^3 1.80 -> 1.88 us). Step, blocks of 128 -> these, us: D3Q27 BGK
// 16^3 2.39 -> 2.14, 28^3 (1.3 blocks per SM) 3.16 -> 2.65, D3Q19 RLBM 28^3 3.5 -> 3.1; from
// 32^3 (1.7) on level or slower, the adjoint already at 28^3 (D3Q27 BGK 4.4 -> 4.75,
// 16^3 3.15 -> 2.8).
constexpr double kStepSpread = 1.7, kAdjointSpread = 1;
template <class L, class Real>
inline Grid latency_grid(const Grid& g, double below) {
  return sizeof(Real) == 8 && L::Q >= 19 && g.bx == kThreads ? spread(g, below, 3) : g;
}

// Whether the loads of a step mark their lines to be evicted first. Each
// population is read once per step, so when the buffers read and written (bytes
// in all) only just exceed the L2 (126 MB), giving up the lines already read
// keeps those being written, which the next step reads. Below that everything
// stays in L2 anyway; above it little does, and the reuse of a line by the
// neighbouring rows suffers. One step in us without and with it: D3Q19 FP64
// BGK 80^3 (156 MB) 23.2 and 17.2, D2Q9 FP64 BGK 1024^2 (151 MB) 22.1 and 15.9,
// D3Q19 FP32 TRT 96^3 (134 MB) 21.8 and 20.2; D3Q19 FP32 TRT 112^3 (214 MB)
// 35.5 and 36.7, 144^3 (454 MB) 71 and 80.
constexpr size_t kL2Bytes = (size_t)126 << 20;
inline bool evict_first_loads(size_t bytes) {
  return bytes > kL2Bytes / 16 * 14 && bytes < kL2Bytes / 16 * 20;
}

struct Span {
  const void* p;
  size_t bytes;
};

inline bool overlaps(Span a, Span b) {
  const uintptr_t a0 = (uintptr_t)a.p, a1 = a0 + a.bytes;
  const uintptr_t b0 = (uintptr_t)b.p, b1 = b0 + b.bytes;
  return a0 < b1 && b0 < a1;
}

// Every written buffer must be disjoint from every other buffer of the call.
template <int NR, int NW>
inline bool any_overlap(const Span (&reads)[NR], const Span (&writes)[NW]) {
  for (int w = 0; w < NW; ++w) {
    for (int r = 0; r < NR; ++r)
      if (overlaps(writes[w], reads[r])) return true;
    for (int v = w + 1; v < NW; ++v)
      if (overlaps(writes[w], writes[v])) return true;
  }
  return false;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

}  // namespace lbcube
