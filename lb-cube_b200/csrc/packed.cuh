// The D3Q27 MRT collision of two FP32 cells in packed arithmetic.
//
// Packed holds the values of two adjacent cells in one 64-bit register pair;
// sm_100a's packed FP32 instructions (add, sub, mul and fma on .f32x2) do two
// operations for one issue slot, each rounded as the scalar one. The step is
// bound by issue slots (1372 instructions per cell one cell at a time), and its
// three 3x3x3 transforms, two thirds of its arithmetic, are sums and exact-product
// FMAs that pack. Ten steps, FP32: 128^3 932 -> 879 us, 200 x 180 x 160 2.57 -> 2.41 ms.
//
// The assembler contracts a packed product and a packed sum of it into one FMA
// whatever -fmad says (observed as different bits), so a product whose sum must
// round twice is never packed: the equilibrium, the relaxation, 3 m_6 and the
// halves stay scalar, and the packed products here feed only FMAs.
#pragma once

#include "collide.cuh"

namespace lbcube {

struct Packed {
  unsigned long long v;
  Packed() = default;
  __device__ __forceinline__ explicit Packed(float both) { asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(both)); }
  __device__ __forceinline__ Packed(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
  __device__ __forceinline__ void lanes(float& a, float& b) const {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  }
};
__device__ __forceinline__ Packed operator+(Packed a, Packed b) {
  Packed r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Packed operator-(Packed a, Packed b) {
  Packed r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Packed fma_rn(Packed a, Packed b, Packed c) {
  Packed r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// fn of each lane, scalar.
template <class Fn>
__device__ __forceinline__ Packed each_lane(Packed x, Fn&& fn) {
  float a, b;
  x.lanes(a, b);
  return Packed(fn(a), fn(b));
}

// div_exact_const<3> of both lanes: the product feeds only FMAs.
__device__ __forceinline__ Packed third(Packed x) {
  const Packed z(1.0f / 3.0f);
  Packed q0;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q0.v) : "l"(x.v), "l"(z.v));
  const Packed r = fma_rn(q0, Packed(-3.0f), x);
  return fma_rn(r, z, q0);
}

__device__ __forceinline__ Packed triple(Packed x) {
  return each_lane(x, [](float a) { return triple(a); });
}

// collide_mrt_d3q27 of the cells f[0] and f[1], bit for bit. Both cells take the
// full expression out of line when either is outside the fast path's bounds,
// and both the IEEE inverse when either has a tiny dividend: each gives the
// fast path's bits wherever that one applies.
__device__ __forceinline__ void collide_mrt_d3q27_pair(float (&f)[2][27], float omega) {
  Packed p[27];
  static_for<27>([&](auto I) { p[LB_I(I)] = Packed(f[0][LB_I(I)], f[1][LB_I(I)]); });
  // macro_state: the same sums in the same order
  Packed density = p[0];
  static_for<26>([&](auto I) { density = density + p[LB_I(I) + 1]; });
  float rho[2], u[2][3];
  density.lanes(rho[0], rho[1]);
  bool fast = bounded27(f[0]) && bounded27(f[1]) && fabsf(rho[0]) <= 0x1p60f && fabsf(rho[1]) <= 0x1p60f &&
              fabsf(omega) <= 0x1p10f;
  static_for<3>([&](auto D) {
    constexpr int d = LB_I(D);
    Packed m(0.0f);
    static_for<27>([&](auto I) {
      constexpr int c = D3Q27::c[LB_I(I)][d];
      if constexpr (c > 0) m = m + p[LB_I(I)];
      if constexpr (c < 0) m = m - p[LB_I(I)];
    });
    float a, b;
    m.lanes(a, b);
    u[0][d] = a / rho[0];
    u[1][d] = b / rho[1];
    fast = fast && fabsf(u[0][d]) <= 0x1p10f && fabsf(u[1][d]) <= 0x1p10f;
  });
  if (!fast) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      // a copy: passing f itself would make it addressable (local memory)
      float fc[27];
      static_for<27>([&](auto K) { fc[LB_I(K)] = f[j][LB_I(K)]; });
      collide_mrt_d3q27_full<float>(fc, omega);
      static_for<27>([&](auto K) { f[j][LB_I(K)] = fc[LB_I(K)]; });
    }
    return;
  }
  Packed m[27], fe[27], eq[27];
  moments_d3q27<Packed, true>(p, m);
  {
    float ea[27], eb[27];
    equilibria<D3Q27>(rho[0], u[0], u_dot_u<D3Q27>(u[0]), ea);
    equilibria<D3Q27>(rho[1], u[1], u_dot_u<D3Q27>(u[1]), eb);
    static_for<27>([&](auto I) { fe[LB_I(I)] = Packed(ea[LB_I(I)], eb[LB_I(I)]); });
  }
  moments_d3q27<Packed, true>(fe, eq);
  static_for<27>([&](auto I) {  // relax_d3q27, its products scalar
    constexpr int i = LB_I(I);
    if constexpr (i >= 4) {
      const float s = rate_d3q27<i>(omega);
      float ma, mb, da, db;
      m[i].lanes(ma, mb);
      (m[i] - eq[i]).lanes(da, db);
      m[i] = Packed(ma - s * da, mb - s * db);
    }
  });
  SafeDividends<float> safe;
  auto see = [&](Packed x) {
    float a, b;
    x.lanes(a, b);
    safe.see(a);
    safe.see(b);
  };
  Packed raw[27];
  moments_to_raw27<Packed>(m, raw);
  see(raw[t27(0, 2, 0)]);
  see(raw[t27(0, 0, 2)]);
  auto half = [](float x) { return 0.5f * x; };
  raw[t27(2, 0, 0)] = third(raw[t27(2, 0, 0)]);
  raw[t27(0, 2, 0)] = each_lane(third(raw[t27(0, 2, 0)]), half);
  raw[t27(0, 0, 2)] = each_lane(third(raw[t27(0, 0, 2)]), half);
  const Packed one_half(0.5f);
  inverse_passes27<Packed>(raw, p, [&](Packed x0, Packed x1, Packed x2, auto last, Packed& fm, Packed& f0, Packed& fp) {
    see(x2);
    Packed q0 = third(x0);
    if constexpr (decltype(last)::value) q0 = Packed(0.0f) + q0;
    const Packed h = each_lane(x1, half);
    const Packed q2 = third(x2);
    fm = fma_rn(one_half, q2, q0 - h);
    f0 = q0 - q2;
    fp = fma_rn(one_half, q2, q0 + h);
  });
  if (!safe.ok()) {
    float mc[2][27];
    static_for<27>([&](auto K) { m[LB_I(K)].lanes(mc[0][LB_I(K)], mc[1][LB_I(K)]); });
    float fa[27], fb[27];
    populations_d3q27_ieee<float>(mc[0], fa);
    populations_d3q27_ieee<float>(mc[1], fb);
    static_for<27>([&](auto K) { p[LB_I(K)] = Packed(fa[LB_I(K)], fb[LB_I(K)]); });
  }
  static_for<27>([&](auto I) { p[LB_I(I)].lanes(f[0][LB_I(I)], f[1][LB_I(I)]); });
}

// Both cells of a pair, packed where that pays.
template <class L, int CT>
__device__ __forceinline__ void collide_pair(float (&f)[2][L::Q], float omega, float omega_minus) {
  if constexpr (L::Q == 27 && CT == kMRT) {
    collide_mrt_d3q27_pair(f, omega);
  } else {
#pragma unroll
    for (int j = 0; j < 2; ++j) collide<L, float, CT>(f[j], omega, omega_minus);
  }
}

}  // namespace lbcube
