// Per-cell collision operators, kept in registers.
//
// Every operator evaluates the same expression tree as LB-Cube's host/device
// physics functions (file:line given per function), so that, compiled without
// FMA contraction (--fmad=false, the engine's build), a step produces the same
// bits as the reference CPU path. Terms whose lattice coefficient is 0 are
// dropped and coefficients of +-1 become additions/subtractions: in IEEE
// arithmetic `x + f*0 == x` and `x + f*(+-1) == x +- f` exactly, so the value
// of every partial sum is unchanged (only the sign of an exact zero can differ).
#pragma once

#include <type_traits>

#include "lattices.cuh"

#define LB_I(I) decltype(I)::value

namespace lbcube {

// exp for the reaction source. The float version is evaluated in double and
// rounded once, which is (almost always) the correctly rounded single-precision
// value that the host libm's expf returns, so the float reaction step tracks
// the CPU path more closely than a single-precision device exp would. The
// argument is -k (B - A): small for any rate that a time step resolves, and
// for |x| < 2^-8 the double value comes from the Taylor polynomial of degree 5
// (Horner, fused multiply-adds): its truncation error x^6 / 720 < 5e-18 is
// below half a unit in the last place of double, so it is as accurate as a
// full double exp for a fraction of the instructions.
template <class Real>
__device__ __forceinline__ Real rexp(Real x);
template <>
__device__ __forceinline__ float rexp<float>(float x) {
  const double d = (double)x;
  if (fabs(d) < 0.00390625) {
    double p = fma(d, 1.0 / 120.0, 1.0 / 24.0);
    p = fma(p, d, 1.0 / 6.0);
    p = fma(p, d, 0.5);
    p = fma(p, d, 1.0);
    return (float)fma(p, d, 1.0);
  }
  return (float)exp(d);
}
template <>
__device__ __forceinline__ double rexp<double>(double x) { return exp(x); }

// Signed sum of velocity components u[d] for the non-zero entries of c_i, in
// ascending d: the value of the dot product c_i . u
// (lattice_physics.hpp:282, :648-652).
template <class L, int i, class Real>
__device__ __forceinline__ Real c_dot(const Real* u) {
  Real s = Real(0);
  bool first = true;
  static_for<L::D>([&](auto D) {
    constexpr int c = L::c[i][LB_I(D)];
    if constexpr (c != 0) {
      const Real t = c > 0 ? u[LB_I(D)] : -u[LB_I(D)];
      s = first ? t : s + t;
      first = false;
    }
  });
  return s;
}

// compute_macro_state (lattice_physics.hpp:227-249): rho = sum f_i in ascending
// i, j_d = sum f_i c_id, u = j / rho.
template <class L, class Real>
__device__ __forceinline__ void macro_state(const Real (&f)[L::Q], Real& rho, Real (&u)[L::D]) {
  Real density = f[0];
  static_for<L::Q - 1>([&](auto I) { density += f[LB_I(I) + 1]; });
  static_for<L::D>([&](auto D) {
    constexpr int d = LB_I(D);
    Real m = Real(0);
    static_for<L::Q>([&](auto I) {
      constexpr int c = L::c[LB_I(I)][d];
      if constexpr (c > 0) m = m + f[LB_I(I)];
      if constexpr (c < 0) m = m - f[LB_I(I)];
    });
    u[d] = m / density;
  });
  // The reference adds f_i * c_id for every i, so a non-finite population
  // makes every velocity component NaN (0 * inf, inf / inf, or a NaN density),
  // while finite populations give exactly the sums above (their zero terms
  // change nothing). Skipping the zero terms loses that, so restore it; a
  // finite density means every population is finite, so the common path only
  // tests the density.
  if (!isfinite(density)) {
    bool bad = false;
    static_for<L::Q>([&](auto I) { bad = bad || !isfinite(f[LB_I(I)]); });
    if (bad) static_for<L::D>([&](auto D) { u[LB_I(D)] = Real(NAN); });
  }
  rho = density;
}

template <class L, class Real>
__device__ __forceinline__ Real u_dot_u(const Real (&u)[L::D]) {
  Real s = u[0] * u[0];
  static_for<L::D - 1>([&](auto D) { s += u[LB_I(D) + 1] * u[LB_I(D) + 1]; });
  return s;
}

// compute_equilibrium (lattice_physics.hpp:267-290):
// w rho (1 + cu/cs2 + cu^2/(2 cs2^2) - u.u/(2 cs2)), grouped as the reference.
template <class L, int i, class Real>
__device__ __forceinline__ Real feq(Real rho, const Real (&u)[L::D], Real usq) {
  constexpr double wd = L::w[i];
  const Real weight = Real(wd);
  const Real inv_cs2 = Real(1.0) / Real(L::cs2);
  const Real cu = c_dot<L, i>(u);
  return weight * rho *
         (Real(1.0) + inv_cs2 * cu + Real(0.5) * inv_cs2 * inv_cs2 * cu * cu -
          Real(0.5) * inv_cs2 * usq);
}

// All Q equilibria of a cell, bit-identical to feq<L, i> for every i but
// computed once per opposite pair: with c_o = -c_i, cu_o = -cu_i exactly, so
// 3 cu_o = -(3 cu_i), 1 + 3 cu_o == 1 - 3 cu_i, and (4.5 cu_o) cu_o ==
// (4.5 cu_i) cu_i, all without rounding differences.
template <class L, class Real>
__device__ __forceinline__ void equilibria(Real rho, const Real (&u)[L::D], Real usq,
                                           Real (&eq)[L::Q]) {
  const Real inv_cs2 = Real(1.0) / Real(L::cs2);
  const Real a = Real(0.5) * inv_cs2 * inv_cs2;  // 4.5, exact
  const Real b = Real(0.5) * inv_cs2;            // 1.5, exact
  const Real tail = b * usq;
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int o = L::opp[i];
    constexpr double wd = L::w[i];
    const Real wr = Real(wd) * rho;
    if constexpr (i == o) {
      eq[i] = wr * (Real(1.0) - tail);  // c_i = 0: 1 + 3*0 + (4.5*0)*0 == 1
    } else if constexpr (i < o) {
      const Real cu = c_dot<L, i>(u);
      const Real p = inv_cs2 * cu;
      const Real t2 = a * cu * cu;
      eq[i] = wr * (Real(1.0) + p + t2 - tail);
      eq[o] = wr * (Real(1.0) - p + t2 - tail);
    }
  });
}

// collide_bgk (lattice_physics.hpp:307-318).
template <class L, class Real>
__device__ __forceinline__ void collide_bgk(Real (&f)[L::Q], Real omega) {
  Real rho, u[L::D], eq[L::Q];
  macro_state<L>(f, rho, u);
  const Real usq = u_dot_u<L>(u);
  equilibria<L>(rho, u, usq, eq);
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    f[i] = f[i] + omega * (eq[i] - f[i]);
  });
}

// compute_omega_minus (lattice_physics.hpp:336-344) with Lambda = 1/4.
template <class Real>
__host__ __device__ inline Real trt_omega_minus(Real omega_plus) {
  const Real magic = Real{1} / Real{4};
  const Real tau_plus = Real{1} / omega_plus;
  const Real tau_minus = magic / (tau_plus - Real{1} / Real{2}) + Real{1} / Real{2};
  return Real{1} / tau_minus;
}

// collide_trt (lattice_physics.hpp:366-398) after compute_macro_state
// (lattice_core.hpp:96-100). omega_minus is precomputed once per launch.
// Evaluated once per opposite pair (i, o): the reference's even parts for i
// and o are the same values, its odd parts exact negatives, so
//   post_i = (f_i - A) - B,  post_o = (f_o - A) + B
// with A = w+ (even - eq_even), B = w- (odd_i - eq_odd_i) reproduces both of
// its results bit for bit. The rest population has odd part +0.
template <class L, class Real>
__device__ __forceinline__ void collide_trt(Real (&f)[L::Q], Real omega_plus, Real omega_minus) {
  Real rho, u[L::D], eq[L::Q];
  macro_state<L>(f, rho, u);
  const Real usq = u_dot_u<L>(u);
  equilibria<L>(rho, u, usq, eq);
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr int o = L::opp[i];
    if constexpr (i == o) {
      f[i] = f[i] - omega_plus * (f[i] - eq[i]);
    } else if constexpr (i < o) {
      const Real even = Real{0.5} * (f[i] + f[o]);
      const Real eq_even = Real{0.5} * (eq[i] + eq[o]);
      const Real odd = Real{0.5} * (f[i] - f[o]);
      const Real eq_odd = Real{0.5} * (eq[i] - eq[o]);
      const Real A = omega_plus * (even - eq_even);
      const Real B = omega_minus * (odd - eq_odd);
      const Real fi = f[i] - A - B;
      const Real fo = f[o] - A + B;
      f[i] = fi;
      f[o] = fo;
    }
  });
}

// ----------------------------------------------------------------------------
// MRT. The forward transforms are written once, generic in the element type,
// with the reference's grouping; instantiated with int at compile time they
// give the integer moment matrix M whose rows are orthogonal, from which the
// inverse M^T D^-1 is taken (coefficient M[r][i] / |M_r|^2).
// ----------------------------------------------------------------------------

// compute_moments_d2q9 (lattice_mrt.hpp:439-455).
template <class T>
__host__ __device__ constexpr void moments_d2q9(const T* f, T* m) {
  m[0] = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8];
  m[1] = -T(4) * f[0] - f[1] - f[2] - f[3] - f[4] + T(2) * (f[5] + f[6] + f[7] + f[8]);
  m[2] = T(4) * f[0] - T(2) * (f[1] + f[2] + f[3] + f[4]) + f[5] + f[6] + f[7] + f[8];
  m[3] = f[1] - f[3] + f[5] - f[6] - f[7] + f[8];
  m[4] = -T(2) * f[1] + T(2) * f[3] + f[5] - f[6] - f[7] + f[8];
  m[5] = f[2] - f[4] + f[5] + f[6] - f[7] - f[8];
  m[6] = -T(2) * f[2] + T(2) * f[4] + f[5] + f[6] - f[7] - f[8];
  m[7] = f[1] - f[2] + f[3] - f[4];
  m[8] = f[5] - f[6] + f[7] - f[8];
}

// compute_moments_d3q19 (lattice_mrt.hpp:617-661).
template <class T>
__host__ __device__ constexpr void moments_d3q19(const T* f, T* m) {
  m[0] = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8] + f[9] + f[10] + f[11] +
         f[12] + f[13] + f[14] + f[15] + f[16] + f[17] + f[18];
  m[1] = -T(30) * f[0] - T(11) * (f[1] + f[2] + f[3] + f[4] + f[5] + f[6]) +
         T(8) * (f[7] + f[8] + f[9] + f[10] + f[11] + f[12] + f[13] + f[14] + f[15] + f[16] +
                 f[17] + f[18]);
  m[2] = T(12) * f[0] - T(4) * (f[1] + f[2] + f[3] + f[4] + f[5] + f[6]) + f[7] + f[8] + f[9] +
         f[10] + f[11] + f[12] + f[13] + f[14] + f[15] + f[16] + f[17] + f[18];
  m[3] = f[1] - f[2] + f[7] - f[8] + f[9] - f[10] + f[11] - f[12] + f[13] - f[14];
  m[4] = -T(4) * f[1] + T(4) * f[2] + f[7] - f[8] + f[9] - f[10] + f[11] - f[12] + f[13] - f[14];
  m[5] = f[3] - f[4] + f[7] + f[8] - f[9] - f[10] + f[15] - f[16] + f[17] - f[18];
  m[6] = -T(4) * f[3] + T(4) * f[4] + f[7] + f[8] - f[9] - f[10] + f[15] - f[16] + f[17] - f[18];
  m[7] = f[5] - f[6] + f[11] + f[12] - f[13] - f[14] + f[15] + f[16] - f[17] - f[18];
  m[8] = -T(4) * f[5] + T(4) * f[6] + f[11] + f[12] - f[13] - f[14] + f[15] + f[16] - f[17] -
         f[18];
  m[9] = T(2) * (f[1] + f[2]) - f[3] - f[4] - f[5] - f[6] + f[7] + f[8] + f[9] + f[10] + f[11] +
         f[12] + f[13] + f[14] - T(2) * (f[15] + f[16] + f[17] + f[18]);
  m[10] = f[3] + f[4] - f[5] - f[6] + f[7] + f[8] + f[9] + f[10] - f[11] - f[12] - f[13] - f[14];
  m[11] = f[7] - f[8] - f[9] + f[10];
  m[12] = f[15] - f[16] - f[17] + f[18];
  m[13] = f[11] - f[12] - f[13] + f[14];
  m[14] = -T(4) * (f[1] + f[2]) + T(2) * (f[3] + f[4] + f[5] + f[6]) + f[7] + f[8] + f[9] +
          f[10] + f[11] + f[12] + f[13] + f[14] - T(2) * (f[15] + f[16] + f[17] + f[18]);
  m[15] = -T(2) * (f[3] + f[4]) + T(2) * (f[5] + f[6]) + f[7] + f[8] + f[9] + f[10] - f[11] -
          f[12] - f[13] - f[14];
  m[16] = f[7] - f[8] + f[9] - f[10] - f[11] + f[12] - f[13] + f[14];
  m[17] = -f[7] - f[8] + f[9] + f[10] + f[15] - f[16] + f[17] - f[18];
  m[18] = f[11] + f[12] - f[13] - f[14] - f[15] - f[16] + f[17] + f[18];
}

template <int Q>
struct MomentMatrix {
  int m[Q][Q];
  int norm[Q];
};

template <int Q, class Fwd>
constexpr MomentMatrix<Q> make_moment_matrix(Fwd fwd) {
  MomentMatrix<Q> r{};
  for (int j = 0; j < Q; ++j) {
    int e[Q] = {};
    int col[Q] = {};
    e[j] = 1;
    fwd(e, col);
    for (int i = 0; i < Q; ++i) r.m[i][j] = col[i];
  }
  for (int i = 0; i < Q; ++i) {
    r.norm[i] = 0;
    for (int j = 0; j < Q; ++j) r.norm[i] += r.m[i][j] * r.m[i][j];
  }
  return r;
}

struct Mrt9 {
  static constexpr MomentMatrix<9> M =
      make_moment_matrix<9>([](const int* f, int* m) { moments_d2q9<int>(f, m); });
  // Order in which compute_populations_d2q9 adds the moment terms (lattice_mrt.hpp:470-534).
  static constexpr int order[9] = {0, 1, 2, 3, 4, 5, 6, 7, 8};
};
struct Mrt19 {
  static constexpr MomentMatrix<19> M =
      make_moment_matrix<19>([](const int* f, int* m) { moments_d3q19<int>(f, m); });
  // Order in which compute_populations_d3q19 adds the moment terms (lattice_mrt.hpp:674-892).
  static constexpr int order[19] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 14, 10, 15, 11, 12, 13, 16, 17, 18};
};

// f_i = sum over r (in the reference's order, zero coefficients skipped) of
// (M[r][i] / |M_r|^2) m_r, evaluated left to right from the first term.
template <class Mx, int Q, class Real>
__device__ __forceinline__ void inverse_orthogonal(const Real (&m)[Q], Real (&f)[Q]) {
  static_for<Q>([&](auto I) {
    constexpr int i = LB_I(I);
    Real acc = Real(0);
    bool first = true;
    static_for<Q>([&](auto K) {
      constexpr int r = Mx::order[LB_I(K)];
      constexpr int coef = Mx::M.m[r][i];
      constexpr int nrm = Mx::M.norm[r];
      if constexpr (coef != 0) {
        // |coef| / |M_r|^2: one product per moment and magnitude, shared by the
        // populations of either sign (-(c m) == (-c) m exactly): the D3Q19 MRT step
        // needs 30 products instead of 50 (FP64, 240 x 355 x 86: 378 -> 352 us)
        const Real term = (Real(coef < 0 ? -coef : coef) / Real(nrm)) * m[r];
        if constexpr (coef > 0) acc = first ? term : acc + term;
        else acc = first ? -term : acc - term;
        first = false;
      }
    });
    f[i] = acc;
  });
}

// collide_mrt_d2q9 (lattice_mrt.hpp:586-603), equilibrium moments (:548-569),
// rates MrtRelaxationRates_D2Q9 (:38-65) with s_nu = omega (lattice_core.hpp:104-107).
template <class Real>
__device__ __forceinline__ void collide_mrt_d2q9(Real (&f)[9], Real omega) {
  Real rho, u[2], m[9];
  macro_state<D2Q9>(f, rho, u);
  moments_d2q9<Real>(f, m);
  const Real ux = u[0], uy = u[1];
  const Real jx = rho * ux, jy = rho * uy;
  const Real usq = ux * ux + uy * uy;
  const Real eq1 = -Real{2} * rho + Real{3} * rho * usq;
  const Real eq2 = rho - Real{3} * rho * usq;
  const Real eq4 = -jx, eq6 = -jy;
  const Real eq7 = rho * (ux * ux - uy * uy);
  const Real eq8 = rho * ux * uy;
  const Real s_e = Real(1.63), s_eps = Real(1.14), s_q = Real(1.92), s_nu = omega;
  m[1] -= s_e * (m[1] - eq1);
  m[2] -= s_eps * (m[2] - eq2);
  m[4] -= s_q * (m[4] - eq4);
  m[6] -= s_q * (m[6] - eq6);
  m[7] -= s_nu * (m[7] - eq7);
  m[8] -= s_nu * (m[8] - eq8);
  inverse_orthogonal<Mrt9>(m, f);
}

// collide_mrt_d3q19 (lattice_mrt.hpp:971-1009) with the equilibrium moments of
// :908-947. Only the shear modes 9-13 use omega; the other non-conserved modes
// relax with the rate 1 the reference hard-wires (:981-1001).
template <class Real>
__device__ __forceinline__ void collide_mrt_d3q19(Real (&f)[19], Real omega) {
  Real rho, u[3], m[19];
  macro_state<D3Q19>(f, rho, u);
  moments_d3q19<Real>(f, m);
  const Real ux = u[0], uy = u[1], uz = u[2];
  const Real jx = rho * ux, jy = rho * uy, jz = rho * uz;
  const Real ux2 = ux * ux, uy2 = uy * uy, uz2 = uz * uz;
  const Real usq = ux2 + uy2 + uz2;
  Real eq[19];
  eq[0] = rho;
  eq[1] = -Real{11} * rho + Real{19} * rho * usq;
  eq[2] = Real{3} * rho - (Real{11} / Real{2}) * rho * usq;
  eq[3] = jx;
  eq[4] = -(Real{2} / Real{3}) * jx;
  eq[5] = jy;
  eq[6] = -(Real{2} / Real{3}) * jy;
  eq[7] = jz;
  eq[8] = -(Real{2} / Real{3}) * jz;
  eq[9] = Real{3} * rho * (Real{2} * ux2 - uy2 - uz2);
  eq[10] = rho * (uy2 - uz2);
  eq[11] = rho * ux * uy;
  eq[12] = rho * uy * uz;
  eq[13] = rho * ux * uz;
  static_for<19>([&](auto I) {
    constexpr int i = LB_I(I);
    if constexpr (i == 0 || i == 3 || i == 5 || i == 7) {
      // conserved: m - 0 * (m - eq) == m
    } else if constexpr (i >= 9 && i <= 13) {
      m[i] -= omega * (m[i] - eq[i]);
    } else if constexpr (i >= 14) {
      m[i] -= Real{1} * (m[i] - Real{0});
    } else {
      m[i] -= Real{1} * (m[i] - eq[i]);
    }
  });
  inverse_orthogonal<Mrt19>(m, f);
}

// D3Q27 orthogonal tensor-product basis (lattice_mrt.hpp:218-426,
// :1023-1305). P0 = 1, P1 = c, P2 = 3c^2 - 2 on c in {-1, 0, 1}, i.e. the
// integer factors below; the separable transforms keep the reference's loop
// order, including the initial `value = 0` of every accumulation.
__host__ __device__ constexpr int p27_basis(int order, int c) {
  return order == 0 ? 1 : (order == 1 ? c : 3 * c * c - 2);
}
__host__ __device__ constexpr int p27_norm(int order) { return order == 0 ? 3 : (order == 1 ? 2 : 6); }
__host__ __device__ constexpr int t27(int a, int b, int c) { return (a * 3 + b) * 3 + c; }

// Position of lattice velocity i in the 3x3x3 tensor layout.
template <int i>
__host__ __device__ constexpr int tensor_slot27() {
  return t27(D3Q27::c[i][0] + 1, D3Q27::c[i][1] + 1, D3Q27::c[i][2] + 1);
}

// a * b + c with one rounding. The D3Q27 transforms use it only where a * b is
// exact (a power of two times b, away from overflow and underflow), so that it
// rounds as the separate product and sum do.
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// One pass of the forward transform along one axis: the sums over c = -1, 0, 1
// of p27_basis(order, c) * p, the reference's accumulation from 0 in ascending
// c. FAST (finite inputs below 2^100, see collide_mrt_d3q27): without the
// leading 0 and the zero-factor term and with the exact product -2 p in the
// FMA: 5 instead of 9 operations per line. Each value is the same real number;
// only the sign of a zero can differ, and the last pass of the inverse
// transform, whose sums start at +0, ends every such difference.
template <class Real, bool FAST>
__device__ __forceinline__ void forward_line27(Real a, Real b, Real c, Real& o0, Real& o1, Real& o2) {
  if constexpr (FAST) {
    o0 = a + b + c;
    o1 = c - a;
    o2 = fma_rn(Real(-2), b, a) + c;
  } else {
    auto sum = [&](auto K) {
      constexpr int k = decltype(K)::value;
      Real v = Real(0);
      v += Real(p27_basis(k, -1)) * a;
      v += Real(p27_basis(k, 0)) * b;
      v += Real(p27_basis(k, 1)) * c;
      return v;
    };
    o0 = sum(std::integral_constant<int, 0>{});
    o1 = sum(std::integral_constant<int, 1>{});
    o2 = sum(std::integral_constant<int, 2>{});
  }
}

// transform_to_moments_d3q27 (lattice_mrt.hpp:1023-1117), one axis after the
// other in the reference's order.
template <class Real, bool FAST = false>
__device__ __forceinline__ void moments_d3q27(const Real (&f)[27], Real (&m)[27]) {
  Real p[27], xt[27], xyt[27], raw[27];
  static_for<27>([&](auto I) { p[tensor_slot27<LB_I(I)>()] = f[LB_I(I)]; });
  static_for<9>([&](auto J) {  // lines along x: (iy, iz)
    constexpr int b = LB_I(J) / 3, c = LB_I(J) % 3;
    forward_line27<Real, FAST>(p[t27(0, b, c)], p[t27(1, b, c)], p[t27(2, b, c)], xt[t27(0, b, c)],
                               xt[t27(1, b, c)], xt[t27(2, b, c)]);
  });
  static_for<9>([&](auto J) {  // along y: (ax, iz)
    constexpr int a = LB_I(J) / 3, c = LB_I(J) % 3;
    forward_line27<Real, FAST>(xt[t27(a, 0, c)], xt[t27(a, 1, c)], xt[t27(a, 2, c)], xyt[t27(a, 0, c)],
                               xyt[t27(a, 1, c)], xyt[t27(a, 2, c)]);
  });
  static_for<9>([&](auto J) {  // along z: (ax, ay)
    constexpr int a = LB_I(J) / 3, b = LB_I(J) % 3;
    forward_line27<Real, FAST>(xyt[t27(a, b, 0)], xyt[t27(a, b, 1)], xyt[t27(a, b, 2)], raw[t27(a, b, 0)],
                               raw[t27(a, b, 1)], raw[t27(a, b, 2)]);
  });
  const Real r200 = raw[t27(2, 0, 0)], r020 = raw[t27(0, 2, 0)], r002 = raw[t27(0, 0, 2)];
  m[0] = raw[t27(0, 0, 0)];
  m[1] = raw[t27(1, 0, 0)];
  m[2] = raw[t27(0, 1, 0)];
  m[3] = raw[t27(0, 0, 1)];
  m[4] = r200 + r020 + r002;
  m[5] = r200 + r200 - r020 - r002;  // 2 r200 exactly
  m[6] = r020 - r002;
  m[7] = raw[t27(1, 1, 0)];
  m[8] = raw[t27(0, 1, 1)];
  m[9] = raw[t27(1, 0, 1)];
  m[10] = raw[t27(2, 1, 0)];
  m[11] = raw[t27(2, 0, 1)];
  m[12] = raw[t27(1, 2, 0)];
  m[13] = raw[t27(0, 2, 1)];
  m[14] = raw[t27(1, 0, 2)];
  m[15] = raw[t27(0, 1, 2)];
  m[16] = raw[t27(1, 1, 1)];
  m[17] = raw[t27(2, 2, 0)];
  m[18] = raw[t27(2, 0, 2)];
  m[19] = raw[t27(0, 2, 2)];
  m[20] = raw[t27(2, 1, 1)];
  m[21] = raw[t27(1, 2, 1)];
  m[22] = raw[t27(1, 1, 2)];
  m[23] = raw[t27(2, 2, 1)];
  m[24] = raw[t27(2, 1, 2)];
  m[25] = raw[t27(1, 2, 2)];
  m[26] = raw[t27(2, 2, 2)];
}

// Correctly rounded x / 3 without a division instruction: Markstein's
// correction step (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990; for divisors
// known in advance, N. Brisebarre, J.-M. Muller, S. K. Raina, IEEE Trans.
// Computers 53(8), 2004):
//   z = RN(1/D),  q0 = RN(x z),  r = x - q0 D (exact with one FMA),  q = RN(q0 + r z).
// With z within half an ulp of 1/D and q0 within one ulp of x / D, q is the
// correctly rounded quotient unless an intermediate value underflows or
// overflows (Markstein's theorem). FP32, against IEEE x / D over every input:
// identical for D = 3 except x = -0 (gives +0) and x = +-inf (gives NaN).
// populations_d3q27 below uses it only where neither can matter (FP64: away
// from the underflow range by a wide margin).
template <int D, class Real>
__device__ __forceinline__ Real div_exact_const(Real x) {
  constexpr Real z = Real(1) / Real(D);
  if constexpr (std::is_same_v<Real, float>) {
    const float q0 = __fmul_rn(x, z);
    const float r = __fmaf_rn(-q0, (float)D, x);
    return __fmaf_rn(r, z, q0);
  } else {
    const double q0 = __dmul_rn(x, z);
    const double r = __fma_rn(-q0, (double)D, x);
    return __fma_rn(r, z, q0);
  }
}

// Running test that every dividend is 0 or at least 2^-123 (FP32) / 2^-960
// (FP64) in magnitude: the unsigned minimum of 2 |bits| - 1, which a zero wraps
// to the largest value (two integer operations per dividend; FP64 on the high
// words, a low word that is not 0 counted in the last bit).
template <class Real>
struct SafeDividends;
template <>
struct SafeDividends<float> {
  unsigned int lo = 0xFFFFFFFFu;
  __device__ __forceinline__ void see(float x) { lo = min(lo, 2u * __float_as_uint(x) - 1u); }
  __device__ __forceinline__ bool ok() const { return lo >= 2u * 0x02000000u - 1u; }  // 2^-123
};
template <>
struct SafeDividends<double> {
  unsigned int lo = 0xFFFFFFFFu;
  __device__ __forceinline__ void see(double x) {
    const unsigned int hi = 2u * (unsigned int)__double2hiint(x) | (__double2loint(x) != 0 ? 1u : 0u);
    lo = min(lo, hi - 1u);
  }
  __device__ __forceinline__ bool ok() const { return lo >= 2u * 0x03F00000u - 1u; }  // 2^-960
};

// transform_to_populations_d3q27 (lattice_mrt.hpp:1130-1225), one axis after
// the other: f(c) = sum over the orders k of (x_k p27_basis(k, c)) / p27_norm(k),
// accumulated from 0 in ascending k.
//
// The reference's form, IEEE divisions and every term. Out of line, so that
// the rare cells that need it keep its divisions out of the kernel's
// instruction stream.
__device__ __forceinline__ float triple(float x) { return 3.0f * x; }
__device__ __forceinline__ double triple(double x) { return 3.0 * x; }
template <class Real>
__device__ __forceinline__ void moments_to_raw27(const Real (&m)[27], Real (&raw)[27]) {
  raw[t27(0, 0, 0)] = m[0];
  raw[t27(1, 0, 0)] = m[1];
  raw[t27(0, 1, 0)] = m[2];
  raw[t27(0, 0, 1)] = m[3];
  raw[t27(2, 0, 0)] = m[4] + m[5];  // times 3, 6 and 6: divided by the callers
  const Real twice = m[4] + m[4] - m[5], thrice = triple(m[6]);
  raw[t27(0, 2, 0)] = twice + thrice;
  raw[t27(0, 0, 2)] = twice - thrice;
  raw[t27(1, 1, 0)] = m[7];
  raw[t27(0, 1, 1)] = m[8];
  raw[t27(1, 0, 1)] = m[9];
  raw[t27(2, 1, 0)] = m[10];
  raw[t27(2, 0, 1)] = m[11];
  raw[t27(1, 2, 0)] = m[12];
  raw[t27(0, 2, 1)] = m[13];
  raw[t27(1, 0, 2)] = m[14];
  raw[t27(0, 1, 2)] = m[15];
  raw[t27(1, 1, 1)] = m[16];
  raw[t27(2, 2, 0)] = m[17];
  raw[t27(2, 0, 2)] = m[18];
  raw[t27(0, 2, 2)] = m[19];
  raw[t27(2, 1, 1)] = m[20];
  raw[t27(1, 2, 1)] = m[21];
  raw[t27(1, 1, 2)] = m[22];
  raw[t27(2, 2, 1)] = m[23];
  raw[t27(2, 1, 2)] = m[24];
  raw[t27(1, 2, 2)] = m[25];
  raw[t27(2, 2, 2)] = m[26];
}

// The three passes of the inverse, `line(x0, x1, x2, first, f-, f0, f+)` giving
// the three populations of one line.
template <class Real, class Line>
__device__ __forceinline__ void inverse_passes27(const Real (&raw)[27], Real (&f)[27], Line&& line) {
  Real zi[27], yzi[27], p[27];
  static_for<9>([&](auto J) {  // along z: (ax, ay)
    constexpr int a = LB_I(J) / 3, b = LB_I(J) % 3;
    line(raw[t27(a, b, 0)], raw[t27(a, b, 1)], raw[t27(a, b, 2)], std::false_type{}, zi[t27(a, b, 0)],
         zi[t27(a, b, 1)], zi[t27(a, b, 2)]);
  });
  static_for<9>([&](auto J) {  // along y: (ax, iz)
    constexpr int a = LB_I(J) / 3, c = LB_I(J) % 3;
    line(zi[t27(a, 0, c)], zi[t27(a, 1, c)], zi[t27(a, 2, c)], std::false_type{}, yzi[t27(a, 0, c)],
         yzi[t27(a, 1, c)], yzi[t27(a, 2, c)]);
  });
  static_for<9>([&](auto J) {  // along x: (iy, iz)
    constexpr int b = LB_I(J) / 3, c = LB_I(J) % 3;
    line(yzi[t27(0, b, c)], yzi[t27(1, b, c)], yzi[t27(2, b, c)], std::true_type{}, p[t27(0, b, c)],
         p[t27(1, b, c)], p[t27(2, b, c)]);
  });
  static_for<27>([&](auto I) { f[LB_I(I)] = p[tensor_slot27<LB_I(I)>()]; });
}

template <class Real>
static __device__ __noinline__ void populations_d3q27_ieee(const Real (&m)[27], Real (&f)[27]) {
  Real raw[27];
  moments_to_raw27<Real>(m, raw);
  raw[t27(2, 0, 0)] = raw[t27(2, 0, 0)] / Real(3);
  raw[t27(0, 2, 0)] = raw[t27(0, 2, 0)] / Real(6);
  raw[t27(0, 0, 2)] = raw[t27(0, 0, 2)] / Real(6);
  inverse_passes27<Real>(raw, f, [](Real x0, Real x1, Real x2, auto, Real& fm, Real& f0, Real& fp) {
    auto sum = [&](auto C) {
      constexpr int c = decltype(C)::value;
      Real v = Real(0);
      v += (x0 * Real(p27_basis(0, c))) / Real(p27_norm(0));
      v += (x1 * Real(p27_basis(1, c))) / Real(p27_norm(1));
      v += (x2 * Real(p27_basis(2, c))) / Real(p27_norm(2));
      return v;
    };
    fm = sum(std::integral_constant<int, -1>{});
    f0 = sum(std::integral_constant<int, 0>{});
    fp = sum(std::integral_constant<int, 1>{});
  });
}

// The fast inverse: 12 operations per line instead of the reference's three
// divisions and nine products and sums. With every moment bounded (the
// caller's guard, so nothing overflows) and every dividend by 6 zero or at
// least 2^-123 (FP64: every dividend at least 2^-960):
//   x0 / 3 and x2 / 3 by div_exact_const; (x1 * +-1) / 2 = +-0.5 x1;
//   x2 / 6 = 0.5 (x2 / 3) exactly, its rounding being that of x2 / 3 scaled by
//   a power of two (the quotient is a normal number), so the sum with it is one
//   FMA with an exact product; (x2 * -2) / 6 = -(x2 / 3).
// The terms whose basis factor is 0 are left out, and the sums start at the
// first term instead of 0 except in the last pass: values are the same, and
// the last pass's +0 start makes every zero result +0, as the reference's is.
// Other cells are recomputed with IEEE divisions.
template <class Real>
__device__ __forceinline__ void populations_d3q27(const Real (&m)[27], Real (&f)[27]) {
  constexpr bool kSingle = std::is_same_v<Real, float>;
  SafeDividends<Real> safe;
  Real raw[27];
  moments_to_raw27<Real>(m, raw);
  if constexpr (!kSingle) safe.see(raw[t27(2, 0, 0)]);
  safe.see(raw[t27(0, 2, 0)]);
  safe.see(raw[t27(0, 0, 2)]);
  raw[t27(2, 0, 0)] = div_exact_const<3>(raw[t27(2, 0, 0)]);
  raw[t27(0, 2, 0)] = Real(0.5) * div_exact_const<3>(raw[t27(0, 2, 0)]);
  raw[t27(0, 0, 2)] = Real(0.5) * div_exact_const<3>(raw[t27(0, 0, 2)]);
  inverse_passes27<Real>(raw, f, [&](Real x0, Real x1, Real x2, auto last, Real& fm, Real& f0, Real& fp) {
    if constexpr (!kSingle) safe.see(x0);
    safe.see(x2);
    Real q0 = div_exact_const<3>(x0);
    if constexpr (decltype(last)::value) q0 = Real(0) + q0;
    const Real h = x1 * Real(0.5);
    const Real q2 = div_exact_const<3>(x2);
    fm = fma_rn(Real(0.5), q2, q0 - h);
    f0 = q0 - q2;
    fp = fma_rn(Real(0.5), q2, q0 + h);
  });
  if (!safe.ok()) {
    // copies: passing m or f itself to the out-of-line call would make them
    // addressable and move them to local memory on the fast path as well
    Real mc[27], fc[27];
    static_for<27>([&](auto K) { mc[LB_I(K)] = m[LB_I(K)]; });
    populations_d3q27_ieee<Real>(mc, fc);
    static_for<27>([&](auto K) { f[LB_I(K)] = fc[LB_I(K)]; });
  }
}

// Projected equilibrium populations of collide_mrt_d3q27 (lattice_mrt.hpp:1242-1268).
template <class Real>
__device__ __forceinline__ void equilibrium_d3q27(Real rho, const Real (&u)[3], Real (&fe)[27]) {
  const Real ux = u[0], uy = u[1], uz = u[2];
  const Real usq = ux * ux + uy * uy + uz * uz;
  static_for<27>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr double wd = D3Q27::w[i];
    const Real cu = c_dot<D3Q27, i>(u);
    fe[i] = Real(wd) * rho * (Real{1} + Real{3} * cu + Real{4.5} * cu * cu - Real{1.5} * usq);
  });
}

// Moment relaxation with MrtRelaxationRates_D3Q27 (lattice_mrt.hpp:161-204).
template <int i, class Real>
__device__ __forceinline__ Real rate_d3q27(Real omega) {
  const Real s_b = Real(1.19), s_e = Real(1.1), s_eps = Real(1.2), s_q = Real(1.2);
  return i == 4 ? s_b : (i <= 9 ? omega : (i <= 15 ? s_e : (i == 16 ? s_eps : s_q)));
}
template <class Real>
__device__ __forceinline__ void relax_d3q27(Real (&m)[27], const Real (&eq)[27], Real omega) {
  static_for<27>([&](auto I) {
    constexpr int i = LB_I(I);
    if constexpr (i >= 4) m[i] -= rate_d3q27<i>(omega) * (m[i] - eq[i]);
  });
}

// The reference's collision term for term, with IEEE divisions: the path of
// every cell that the guard of collide_mrt_d3q27 sends away. Out of line, so
// its code stays out of the kernel's instruction stream.
template <class Real>
static __device__ __noinline__ void collide_mrt_d3q27_full(Real (&f)[27], Real omega) {
  Real rho, u[3], m[27], fe[27], eq[27];
  macro_state<D3Q27>(f, rho, u);
  moments_d3q27<Real>(f, m);
  equilibrium_d3q27<Real>(rho, u, fe);
  moments_d3q27<Real>(fe, eq);
  relax_d3q27<Real>(m, eq, omega);
  populations_d3q27_ieee<Real>(m, f);
}

// Largest magnitude of the 27 populations below 2^60 (false for infinities;
// NaN is the density's business). FP64: on the high words.
__device__ __forceinline__ bool bounded27(const float (&f)[27]) {
  float m = 0.0f;
  static_for<27>([&](auto K) { m = fmaxf(m, fabsf(f[LB_I(K)])); });
  return m < 0x1p60f;
}
__device__ __forceinline__ bool bounded27(const double (&f)[27]) {
  unsigned int m = 0;
  static_for<27>([&](auto K) { m = max(m, 2u * (unsigned int)__double2hiint(f[LB_I(K)])); });
  return m < 2u * 0x43B00000u;
}

// collide_mrt_d3q27 (lattice_mrt.hpp:1284-1305) with the projected
// equilibrium of :1242-1268 and MrtRelaxationRates_D3Q27 (:161-204).
// Guard: every |f_i| < 2^60, |rho| <= 2^60, every |u_d| <= 2^10 and |omega| <=
// 2^10 (false for NaN). The equilibrium populations are then below 2^86, both
// sets of moments below 2^100 and the relaxed ones below 2^110, so every value
// of the transforms is finite and far from overflow, which is what the fast
// transforms need; the equilibrium may be formed per opposite pair. Other
// cells run the full expression out of line.
//
// Bound by its instructions, not its bytes (216 B per FP32 cell). Counting the
// arithmetic: 5 + 5 + 12 operations per line of the three transforms (27 lines
// each) against 9 + 9 + 18 before. FP32 128^3: 113.5 -> 101.0 us per step (4.0 ->
// 4.5 TB/s of the 6.6 a copy moves).
template <class Real>
__device__ __forceinline__ void collide_mrt_d3q27(Real (&f)[27], Real omega) {
  Real rho, u[3];
  macro_state<D3Q27>(f, rho, u);
  const bool fast = bounded27(f) && fabs(rho) <= Real(0x1p60) && fabs(u[0]) <= Real(0x1p10) &&
                    fabs(u[1]) <= Real(0x1p10) && fabs(u[2]) <= Real(0x1p10) &&
                    fabs(omega) <= Real(0x1p10);
  if (!fast) {
    // a copy: passing f itself would make it addressable (local memory)
    Real fc[27];
    static_for<27>([&](auto K) { fc[LB_I(K)] = f[LB_I(K)]; });
    collide_mrt_d3q27_full<Real>(fc, omega);
    static_for<27>([&](auto K) { f[LB_I(K)] = fc[LB_I(K)]; });
    return;
  }
  Real m[27], fe[27], eq[27];
  moments_d3q27<Real, true>(f, m);
  equilibria<D3Q27>(rho, u, u_dot_u<D3Q27>(u), fe);
  moments_d3q27<Real, true>(fe, eq);
  relax_d3q27<Real>(m, eq, omega);
  populations_d3q27<Real>(m, f);
}

// ----------------------------------------------------------------------------
// Regularized (RLBM) collision, collide_regularized (lattice_physics.hpp:422-605)
// with compute_pi_neq_* (:116-211).
// ----------------------------------------------------------------------------
template <class L, class Real>
__device__ __forceinline__ void collide_rlbm(Real (&f)[L::Q], Real omega) {
  Real rho, u[L::D], fe[L::Q];
  macro_state<L>(f, rho, u);
  const Real usq = u_dot_u<L>(u);
  equilibria<L>(rho, u, usq, fe);
  const Real hp = Real{9} / Real{2};
  const Real cs2 = Real(L::cs2);
  // Pi_neq = sum_i (f_i - feq_i) c_i c_i, accumulated from zero in ascending i.
  Real pxx = Real(0), pyy = Real(0), pzz = Real(0), pxy = Real(0), pxz = Real(0), pyz = Real(0);
  static_for<L::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    const Real fn = f[i] - fe[i];
    constexpr int ix = L::c[i][0], iy = L::c[i][1], iz = L::c[i][2];
    const Real cx = Real(ix), cy = Real(iy), cz = Real(iz);
    (void)cz;
    pxx += fn * cx * cx;
    pyy += fn * cy * cy;
    pxy += fn * cx * cy;
    if constexpr (L::D == 3) {
      pzz += fn * cz * cz;
      pxz += fn * cx * cz;
      pyz += fn * cy * cz;
    }
  });
  if constexpr (L::id == kD2Q9) {
    const Real ux = u[0], uy = u[1];
    const Real a_xxx = Real{3} * ux * pxx;
    const Real a_yyy = Real{3} * uy * pyy;
    const Real a_xxy = Real{2} * ux * pxy + uy * pxx;
    const Real a_xyy = Real{2} * uy * pxy + ux * pyy;
    static_for<9>([&](auto I) {
      constexpr int i = LB_I(I);
      constexpr double wd = L::w[i];
      constexpr int ix = L::c[i][0], iy = L::c[i][1];
      const Real cx = Real(ix), cy = Real(iy);
      const Real q_xx = cx * cx - cs2, q_yy = cy * cy - cs2, q_xy = cx * cy;
      const Real second = q_xx * pxx + q_yy * pyy + Real{2} * q_xy * pxy;
      const Real h_xxx = cx * cx * cx - Real{3} * cs2 * cx;
      const Real h_yyy = cy * cy * cy - Real{3} * cs2 * cy;
      const Real h_xxy = cx * cx * cy - cs2 * cy;
      const Real h_xyy = cx * cy * cy - cs2 * cx;
      const Real third = a_xxx * h_xxx + a_yyy * h_yyy + Real{3} * (a_xxy * h_xxy + a_xyy * h_xyy);
      const Real rec = Real(wd) * hp * (second + third);
      f[i] = fe[i] + (Real{1} - omega) * rec;
    });
  } else {
    const Real ux = u[0], uy = u[1], uz = u[2];
    const Real a_xxx = Real{3} * ux * pxx;
    const Real a_yyy = Real{3} * uy * pyy;
    const Real a_zzz = Real{3} * uz * pzz;
    const Real a_xxy = Real{2} * ux * pxy + uy * pxx;
    const Real a_xxz = Real{2} * ux * pxz + uz * pxx;
    const Real a_yyz = Real{2} * uy * pyz + uz * pyy;
    Real a_xyy, a_xzz, a_yzz, a_xyz;
    if constexpr (L::id == kD3Q19) {
      a_xyy = Real{2} * uy * pxy + ux * pyy;
      a_xzz = Real{2} * uz * pxz + ux * pzz;
      a_yzz = Real{2} * uz * pyz + uy * pzz;
      a_xyz = Real(0);
    } else {
      a_xyy = ux * pyy + Real{2} * uy * pxy;
      a_xzz = ux * pzz + Real{2} * uz * pxz;
      a_yzz = uy * pzz + Real{2} * uz * pyz;
      a_xyz = ux * pyz + uy * pxz + uz * pxy;
    }
    static_for<L::Q>([&](auto I) {
      constexpr int i = LB_I(I);
      constexpr double wd = L::w[i];
      constexpr int ix = L::c[i][0], iy = L::c[i][1], iz = L::c[i][2];
    const Real cx = Real(ix), cy = Real(iy), cz = Real(iz);
      const Real q_xx = cx * cx - cs2, q_yy = cy * cy - cs2, q_zz = cz * cz - cs2;
      const Real q_xy = cx * cy, q_xz = cx * cz, q_yz = cy * cz;
      const Real second = q_xx * pxx + q_yy * pyy + q_zz * pzz +
                          Real{2} * (q_xy * pxy + q_xz * pxz + q_yz * pyz);
      const Real h_xxx = cx * cx * cx - Real{3} * cs2 * cx;
      const Real h_yyy = cy * cy * cy - Real{3} * cs2 * cy;
      const Real h_zzz = cz * cz * cz - Real{3} * cs2 * cz;
      const Real h_xxy = cx * cx * cy - cs2 * cy;
      const Real h_xxz = cx * cx * cz - cs2 * cz;
      const Real h_xyy = cx * cy * cy - cs2 * cx;
      const Real h_yyz = cy * cy * cz - cs2 * cz;
      const Real h_xzz = cx * cz * cz - cs2 * cx;
      const Real h_yzz = cy * cz * cz - cs2 * cy;
      const Real h_xyz = cx * cy * cz;
      (void)h_xxx, (void)h_yyy, (void)h_zzz, (void)h_xyz;  // unused by the D3Q19 branch
      Real third;
      if constexpr (L::id == kD3Q19) {
        third = Real{3} * (h_xxy + h_yzz) * (a_xxy + a_yzz) + (h_xxy - h_yzz) * (a_xxy - a_yzz) +
                Real{3} * (h_xzz + h_xyy) * (a_xzz + a_xyy) + (h_xzz - h_xyy) * (a_xzz - a_xyy) +
                Real{3} * (h_yyz + h_xxz) * (a_yyz + a_xxz) + (h_yyz - h_xxz) * (a_yyz - a_xxz);
      } else {
        third = a_xxx * h_xxx + a_yyy * h_yyy + a_zzz * h_zzz +
                Real{3} * (a_xxy * h_xxy + a_xxz * h_xxz + a_xyy * h_xyy + a_yyz * h_yyz +
                           a_xzz * h_xzz + a_yzz * h_yzz) +
                Real{6} * a_xyz * h_xyz;
      }
      const Real rec = Real(wd) * hp * (second + third);
      f[i] = fe[i] + (Real{1} - omega) * rec;
    });
  }
}

// collide_cell dispatch (lattice_core.hpp:90-126, lattice_cuda.cu:90-126).
template <class L, class Real, int CT>
__device__ __forceinline__ void collide(Real (&f)[L::Q], Real omega, Real omega_minus) {
  if constexpr (CT == kBGK) {
    collide_bgk<L>(f, omega);
  } else if constexpr (CT == kTRT) {
    collide_trt<L>(f, omega, omega_minus);
  } else if constexpr (CT == kMRT) {
    if constexpr (L::id == kD2Q9) collide_mrt_d2q9<Real>(f, omega);
    else if constexpr (L::id == kD3Q19) collide_mrt_d3q19<Real>(f, omega);
    else collide_mrt_d3q27<Real>(f, omega);
  } else {
    collide_rlbm<L>(f, omega);
  }
}

// ----------------------------------------------------------------------------
// Advection-diffusion (lattice_physics.hpp:607-743).
// ----------------------------------------------------------------------------

// compute_concentration: C = sum g_i in ascending i.
template <class S, class Real>
__device__ __forceinline__ Real concentration(const Real (&g)[S::Q]) {
  Real c = g[0];
  static_for<S::Q - 1>([&](auto I) { c += g[LB_I(I) + 1]; });
  return c;
}

// compute_scalar_equilibrium: w C (1 + (c.u) / cs2), with a true division by cs2.
template <class S, int i, class Real>
__device__ __forceinline__ Real geq(Real conc, const Real (&u)[S::D]) {
  constexpr double wd = S::w[i];
  const Real cu = c_dot<S, i>(u);
  const Real cs2 = Real(S::cs2);
  return Real(wd) * conc * (Real(1.0) + cu / cs2);
}

// collide_scalar_bgk: g_i += omega_c (g_eq - g_i) + w_i S.
template <class S, class Real>
__device__ __forceinline__ void collide_scalar(Real (&g)[S::Q], const Real (&u)[S::D], Real omega_c,
                                               Real source) {
  const Real conc = concentration<S>(g);
  static_for<S::Q>([&](auto I) {
    constexpr int i = LB_I(I);
    constexpr double wd = S::w[i];
    const Real eq = geq<S, i>(conc, u);
    g[i] += omega_c * (eq - g[i]) + Real(wd) * source;
  });
}

template <class Real> struct RealEps;
template <> struct RealEps<float> { static constexpr float value = 1.1920928955078125e-07f; };
template <> struct RealEps<double> { static constexpr double value = 2.220446049250313080847e-16; };

// compute_reaction_ab_source: exact one-step A + B -> C batch solution; the
// returned increment is applied to both species.
template <class Real>
__device__ __forceinline__ Real reaction_source(Real a, Real b, Real k) {
  const Real abs_a = a < Real{} ? -a : a;
  const Real abs_b = b < Real{} ? -b : b;
  const Real diff = b - a;
  const Real abs_diff = diff < Real{} ? -diff : diff;
  const Real tol = Real(64.0) * RealEps<Real>::value * (Real(1.0) + abs_a + abs_b);
  Real a_after;
  if (abs_diff <= tol) {
    a_after = a / (Real(1.0) + k * a);
  } else {
    const Real att = rexp<Real>(-k * diff);
    a_after = a * diff * att / (b - a * att);
  }
  return a_after - a;
}

// Two species pulled, one exact A+B->C source applied to both
// (lattice_core.hpp:403-411).
template <class SL, class Real>
__device__ __forceinline__ void react_pair(Real (&a)[SL::Q], Real (&b)[SL::Q],
                                           const Real (&u)[SL::D], Real omega_c, Real k) {
  const Real ca = concentration<SL>(a);
  const Real cb = concentration<SL>(b);
  const Real src = reaction_source<Real>(ca, cb, k);
  collide_scalar<SL>(a, u, omega_c, src);
  collide_scalar<SL>(b, u, omega_c, src);
}

}  // namespace lbcube
