// gd_fft_reg.cuh -- register-resident phi transforms: small DFTs of any 2/3/5
// composite length with compile-time roots, and the split of a row length
// N = T A B over a team of 2 T threads (gd_fused_reg.cuh).
#pragma once

#include "gd_fft_core.cuh"

namespace gd {

// cos and sin of 2 pi num / den at compile time (Taylor series after reduction
// to an eighth turn; the terms left out are below 1e-20).
struct CRoot {
  double c, s;
};
constexpr CRoot c_root(long num, long den) {
  num %= den;
  if (num < 0) num += den;
  // octant: 8 num / den, remainder angle in [0, pi / 4]
  const long oct = 8 * num / den;
  const long rem8 = 8 * num - oct * den;  // angle = 2 pi (oct / 8) + 2 pi rem8 / (8 den)
  const double pi = 3.14159265358979323846;
  const bool odd = oct & 1;
  const double x = odd ? 2.0 * pi * (double)(den - rem8) / (8.0 * (double)den)
                       : 2.0 * pi * (double)rem8 / (8.0 * (double)den);
  double c = 1.0, s = x, tc = 1.0, ts = x;
  for (int k = 1; k < 14; ++k) {
    tc *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
    ts *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
    c += tc;
    s += ts;
  }
  // odd octants measure the angle back from the next multiple of pi / 2... in quarter turns:
  const long q = (oct + (odd ? 1 : 0)) / 2;  // nearest quarter turn
  const double rs = odd ? -s : s;
  switch (q % 4) {
    case 0: return CRoot{c, rs};
    case 1: return CRoot{-rs, c};
    case 2: return CRoot{-c, -rs};
    default: return CRoot{rs, -c};
  }
}

// a * exp(-2 pi i NUM / DEN)
template <long NUM, long DEN, typename C>
__device__ __forceinline__ C mul_root(C a) {
  typedef decltype(a.x) S;
  constexpr long n = ((NUM % DEN) + DEN) % DEN;
  if constexpr (4 * n == DEN) {
    C r; r.x = a.y; r.y = -a.x;
    return r;
  } else if constexpr (2 * n == DEN) {
    C r; r.x = -a.x; r.y = -a.y;
    return r;
  } else if constexpr (4 * n == 3 * DEN) {
    C r; r.x = -a.y; r.y = a.x;
    return r;
  } else if constexpr (n != 0) {
    constexpr CRoot w = c_root(n, DEN);
    constexpr S c = (S)w.c, s = (S)w.s;
    C r; r.x = a.x * c + a.y * s; r.y = a.y * c - a.x * s;
    return r;
  } else {
    return a;
  }
}

// In-register DFT of R points, natural order in and out: the radices of
// gd_fft_core.cuh, and composites R = R1 R2 by one Cooley-Tukey step
//   X[k1 + R1 k2] = sum_n2 W_R^(n2 k1) W_R2^(n2 k2) sum_n1 x[R2 n1 + n2] W_R1^(n1 k1).
template <int R> struct RSplit { static constexpr int r1 = 1; };
template <> struct RSplit<6> { static constexpr int r1 = 2; };
template <> struct RSplit<9> { static constexpr int r1 = 3; };
template <> struct RSplit<10> { static constexpr int r1 = 2; };
template <> struct RSplit<12> { static constexpr int r1 = 3; };
template <> struct RSplit<15> { static constexpr int r1 = 3; };
template <> struct RSplit<18> { static constexpr int r1 = 3; };
template <> struct RSplit<20> { static constexpr int r1 = 5; };
template <> struct RSplit<24> { static constexpr int r1 = 3; };
template <> struct RSplit<25> { static constexpr int r1 = 5; };
template <> struct RSplit<30> { static constexpr int r1 = 5; };
template <> struct RSplit<32> { static constexpr int r1 = 2; };

template <int R, typename C> struct RDft;

template <int R, int R1, int R2, int N2, int K1, typename C>
__device__ __forceinline__ void rdft_twiddle(C* t) {
  if constexpr (K1 < R1) {
    t[K1] = mul_root<(long)N2 * K1, R>(t[K1]);
    rdft_twiddle<R, R1, R2, N2, K1 + 1, C>(t);
  }
}
template <int R, int R1, int R2, int N2, typename C>
__device__ __forceinline__ void rdft_first(C* v) {
  if constexpr (N2 < R2) {
    C t[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + N2];
    RDft<R1, C>::run(t);
    rdft_twiddle<R, R1, R2, N2, 0, C>(t);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) v[R2 * n1 + N2] = t[n1];
    rdft_first<R, R1, R2, N2 + 1, C>(v);
  }
}
template <int R, typename C> struct RDft {
  static __device__ __forceinline__ void run(C* v) {
    constexpr int R1 = RSplit<R>::r1;
    if constexpr (R == 1) {
      return;
    } else if constexpr (R1 == 1) {
      Dft<R, C>::run(v);
    } else {
      constexpr int R2 = R / R1;
      rdft_first<R, R1, R2, 0, C>(v);
      C o[R];
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        C t[R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) t[n2] = v[R2 * k1 + n2];
        RDft<R2, C>::run(t);
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) o[k1 + R1 * k2] = t[k2];
      }
#pragma unroll
      for (int k = 0; k < R; ++k) v[k] = o[k];
    }
  }
};

}  // namespace gd
