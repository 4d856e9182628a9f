// The storage policies of shifted 16-bit populations: how a pair of codes is
// decoded into FP32 values, collided and encoded.
//   ShiftedStorage<fmt>  decoded to populations f
//   DevStorage<fmt>      collided as the stored deviations
#pragma once

#include "collide.cuh"
#include "collide_dev.cuh"

namespace lbcube {

// Shifted 16-bit storage of LB populations: the stored code h_i stands for
//   v_i = S (f_i / w_i - rho0)      (the codec of each format, collide_dev.cuh)
// so f_i = w_i (rho0 + v_i / S). Subtracting the rest state w_i rho0 keeps
// only the small deviation (a few 1e-2 of w_i at Mach 0.1), dividing by w_i
// puts every direction on the same scale, and S places that range where the
// format resolves it best. This policy decodes to f and runs the reference
// collision (MRT, RLBM, conversions); DevStorage below collides on v directly.
template <int FMT>
struct ShiftedStorage {
  using elem = unsigned short;
  static constexpr bool kDecoded = true;
  struct Params {
    float rho0;
  };
  template <class L, int i>
  __device__ __forceinline__ static float decode(elem h, const Params& p) {
    constexpr double wd = L::w[i];
    return float(wd) * fmaf(Codec<FMT>::decode(h), 1.0f / Codec<FMT>::S, p.rho0);
  }
  template <class L, int i>
  __device__ __forceinline__ static elem encode(float f, const Params& p) {
    constexpr double wd = L::w[i];
    return Codec<FMT>::encode((f * float(1.0 / wd) - p.rho0) * Codec<FMT>::S);
  }
  template <class L, int i>
  __device__ __forceinline__ static float2 decode_pair(unsigned int w, const Params& p) {
    return make_float2(decode<L, i>((elem)w, p), decode<L, i>((elem)(w >> 16), p));
  }
  template <class L, int i>
  __device__ __forceinline__ static unsigned int encode_pair(float a, float b, const Params& p) {
    return __byte_perm(encode<L, i>(a, p), encode<L, i>(b, p), 0x5410);
  }
  template <class L, int CT>
  __device__ __forceinline__ static void collide_cell(float (&f)[L::Q], float omega, float omega_minus,
                                                      const Params&) {
    collide<L, float, CT>(f, omega, omega_minus);
  }
};

// 16-bit storage whose collision runs on the stored deviations (BGK, TRT, and
// the D2Q9 / D3Q19 MRT).
template <int FMT>
struct DevStorage {
  using elem = unsigned short;
  static constexpr bool kDecoded = false;
  struct Params {
    float rho0;
  };
  template <class L, int i>
  __device__ __forceinline__ static float2 decode_pair(unsigned int w, const Params&) {
    return Codec<FMT>::decode2(w);
  }
  template <class L, int i>
  __device__ __forceinline__ static unsigned int encode_pair(float a, float b, const Params&) {
    return Codec<FMT>::encode2(a, b);
  }
  template <class L, int CT>
  __device__ __forceinline__ static void collide_cell(float (&v)[L::Q], float omega, float omega_minus,
                                                      const Params& p) {
    static_assert(CT == kBGK || CT == kTRT || (CT == kMRT && L::Q != 27),
                  "deviation-space collision is BGK, TRT, or D2Q9 / D3Q19 MRT");
    if constexpr (CT == kMRT) collide_dev_mrt<L, FMT>(v, omega, p.rho0);
    else collide_dev<L, CT, FMT>(v, omega, omega_minus, p.rho0);
  }
};

}  // namespace lbcube
