// Test helper: answers questions about the host side of the kernels' launch rules,
// one per line of standard input, from the engine's own headers.
//   div n d            n / d through FastDiv
//   grid nx ny nz      per grid (plain, statistics, FP64 3-D): threads per block, blocks per plane, blocks
//                      launched; then the partials contract
//   fluid L OP DIAG nx ny nz    1 if the FP32 fluid step takes two cells per thread
//   adjoint L OP nx ny nz       the same for the FP32 adjoint step
//   coupled L FMT RESIDENT nx ny nz    1 if the 16-bit coupled step takes four
// (L: 9, 19 or 27; OP: 0 BGK, 1 TRT, 2 MRT, 3 RLBM; FMT: 0 FP16, 1 BF16, 2 E3M12, 3 Q15; RESIDENT: blocks of its one-cell kernel per SM)
#include <cstdio>
#include <cstring>

#include "../lb-cube_b200/csrc/adjoint.cuh"
#include "../lb-cube_b200/csrc/step_cell.cuh"
#include "../lb-cube_b200/csrc/stream_codes.cuh"

using namespace lbcube;

template <class L, int OP, bool DIAG>
int fluid(const Grid& g) {
  return kUsePairs<L, float, DIAG> && pairs_eligible<DIAG>(g, kPairRule<L, OP>, (float*)0x100);
}
template <class L>
int fluid_of(int op, int diag, const Grid& g) {
  const int v[4][2] = {{fluid<L, 0, false>(g), fluid<L, 0, true>(g)}, {fluid<L, 1, false>(g), fluid<L, 1, true>(g)},
                       {fluid<L, 2, false>(g), fluid<L, 2, true>(g)}, {fluid<L, 3, false>(g), fluid<L, 3, true>(g)}};
  return v[op][diag];
}
template <class L>
int adjoint_of(int op, const Grid& g) {
  const float* p = (const float*)0x100;
  return op == 0   ? pairs_eligible<true>(g, kAdjointPairRule<L, 0>, p)
         : op == 1 ? pairs_eligible<true>(g, kAdjointPairRule<L, 1>, p)
                   : pairs_eligible<true>(g, kAdjointPairRule<L, 2>, p);
}
template <class L>
int coupled_of(int fmt, int resident, const Grid& g) {
  const CellRule r = fmt == kF16S    ? coupled_codes_rule<L, kF16S>(resident)
                     : fmt == kBF16S ? coupled_codes_rule<L, kBF16S>(resident)
                                     : coupled_codes_rule<L, kQ15S>(resident);
  return g.nx % kCodeCells == 0 && several_cells_pay(g.nx, g.ny, g.nz, kCodeCells, kThreads, r);
}

int main() {
  char what[16];
  while (scanf("%15s", what) == 1) {
    if (strcmp(what, "div") == 0) {
      unsigned n, d;
      if (scanf("%u %u", &n, &d) != 2) return 2;
      printf("%u\n", FastDiv(d)(n));
      continue;
    }
    int a[3];
    size_t n[3];
    const int extra = strcmp(what, "grid") == 0 ? 0 : strcmp(what, "adjoint") == 0 ? 2 : 3;
    for (int i = 0; i < extra; ++i)
      if (scanf("%d", &a[i]) != 1) return 2;
    if (scanf("%zu %zu %zu", &n[0], &n[1], &n[2]) != 3) return 2;
    Grid g{};
    if (validate_domain(false, 1, 1, 1, n[2] == 1 ? 2 : 3, n[0], n[1], n[2], g) != cudaSuccess) return 3;
    if (extra == 0) {
      for (const Grid& v : {g, stats_grid(g), latency_grid<D3Q19, double>(g, kStepSpread)}) printf("%d %d %lld ", v.bx, v.tiles, v.launched());
      printf("%lld\n", g.blocks());
    } else if (extra == 2) printf("%d\n", a[0] == 9 ? adjoint_of<D2Q9>(a[1], g) : adjoint_of<D3Q19>(a[1], g));
    else if (strcmp(what, "fluid") == 0)
      printf("%d\n", a[0] == 9    ? fluid_of<D2Q9>(a[1], a[2], g)
                     : a[0] == 19 ? fluid_of<D3Q19>(a[1], a[2], g)
                                  : fluid_of<D3Q27>(a[1], a[2], g));
    else printf("%d\n", a[0] == 9 ? coupled_of<D2Q9>(a[1], a[2], g) : coupled_of<D3Q19>(a[1], a[2], g));
  }
  return 0;
}
