// gd_fused_reg.cuh -- the nonlinear phases of the mixed-precision step on
// register-resident phi transforms (the runtime-length form is in gd_fused.cu).
//
// A team of 2 T threads owns one (shell, block of two colatitude pairs) from
// the Fourier coefficients to the folded transforms of the products: thread
// (j, ii) = (team lane / 2, team lane % 2) works on pair ii.  The row length is
// N = T A B.  Inverse transform of a component (frequencies k = j + T (r + B s)):
//   1. thread j: DFT over s (A points) and r (B points) in registers -> index
//      u = A q + a, times W_N^(j u);
//   2. one exchange through shared memory per a (T x B elements);
//   3. thread t: for q = t + T w the DFT over j (T points) -> longitude
//      phi = A q + a + A B p, p = 0 .. T - 1.
// The thread then holds A B longitudes of its pair, multiplies and accumulates
// them in registers, and the forward transform of the sum runs the three steps
// backwards (T points over p, exchange, B points over q, A points over a).
//
// What bounds it: two warps per scheduler (the sums, the held spectrum and a
// DFT fill 255 registers at N = 768) against shared-memory latency; issue ~45%,
// FP32 pipe ~50%, shared memory ~50%.  Against radix passes of a whole CTA
// through shared memory with the sums kept there (47 k warp instructions per
// team and ten transforms, now 17 k, ncu) it has one exchange instead of three
// passes, no block barrier, no index arithmetic (every address is a thread base
// plus a constant), no read-modify-write of the sums, and packed FP32 adds.
// The exchange rows have an odd stride, so both its sides are free of bank
// conflicts; the next component's coefficients (one contiguous run) arrive by
// cp.async while the current one is transformed; CTAs are persistent, so the
// tables are filled once.  Measured (B200, before -> after): velocity /
// temperature / induction phase at lmax 255, nlon 768, nr 129: 839 / 437 / 414
// -> 419 / 258 / 258 us; lmax 341, nlon 1024, nr 33: 1138 / 707 / 605 -> 225 /
// 146 / 148 us; lmax 127, nlon 256, nr 65: 127 / 83 / 76 -> 33 / 24 / 24 us.
// Reading the spectrum again for each a instead of holding it allows 12 warps
// at 168 registers but makes shared memory the limit (79%): 416 / 248 us for
// velocity / induction, no better; holding half of it spills.
//
// SPLIT (A = 3 and M < N / 3, the 3/2 rule): frequencies N/3 <= k < 2N/3 carry
// nothing, so the middle input of the 3-point step is dropped in the inverse
// transform and its middle output never formed in the forward one.
#pragma once

#include <type_traits>

#include "gd_fft_reg.cuh"
#include "gd_fused.cuh"

namespace gd {

template <int T_, int A_, int B_> struct RowPlan {
  static constexpr int T = T_, A = A_, B = B_, K = A_ * B_, N = T_ * A_ * B_, W = B_ / T_;
  static_assert(B_ % T_ == 0 && K % 2 == 0 && (T_ <= 16 || T_ == 32), "row plan");
  static constexpr int TEAM = 2 * T;
  static constexpr int TPW = TEAM <= 32 ? 32 / TEAM : 1;        // teams per warp
  static constexpr int WPT = TEAM <= 32 ? 1 : TEAM / 32;        // warps per team
  static constexpr int SB = B | 1;                              // exchange row stride
  static constexpr int RO = (T * SB + 7) / 16 * 16 + 8;         // pair ii at ii RO: the two pairs on disjoint banks
};

template <class PL, bool SPLIT, int PH>
struct FusedRegGeom {
  static constexpr int ROWS = SPLIT ? PL::N / 3 + 1 : PL::N / 2 + 1;  // orders of the input stage, zero past M
  // components whose spectrum stays in registers while its sub-transforms run
  static constexpr bool HOLD = SPLIT || PL::K <= 40;
  static constexpr int STAGES = HOLD ? 1 : 2;
  static constexpr int IN = ROWS * 2;                                  // float4 per stage
  // float2 per exchange buffer, which also takes the mirrored orders of both pairs
  static constexpr int EX0 = PL::RO > ROWS ? 2 * PL::RO : 2 * ROWS;
  static constexpr int EX = (EX0 + 15) / 16 * 16 + (PL::T == 4 ? 4 : 0);
  static constexpr size_t team_bytes_x(int xbuf) {
    return (size_t)STAGES * IN * sizeof(float4) + (size_t)xbuf * EX * sizeof(float2) +
           (PH == FUSED_TEMPERATURE ? (size_t)PL::K * PL::TEAM * sizeof(float2) : 0);
  }
  static constexpr size_t cta_bytes() {  // roots and longitude factors
    return ((size_t)(PL::K * (PL::T + 1) + (PH == FUSED_VELOCITY ? (PL::N + 1) / 2 : 0)) * sizeof(float2) + 15) / 16 * 16;
  }
  // Registers of a thread: the sums (2 K), the held spectrum, a B- or T-point
  // DFT, ~40 more.  One CTA of 8 warps on an SM at 255 registers, else CTAs of 4 warps.
  static constexpr int REGS = 2 * PL::K + (SPLIT ? 4 * PL::B : HOLD ? 2 * PL::K : 64) + 2 * (PL::B > PL::T ? PL::B : PL::T) + 40;
  static constexpr int MINB = REGS > 168 ? 1 : REGS > 128 ? 3 : 4;
  static constexpr size_t LIMIT = (size_t)227 * 1024 / MINB - 1024;
  static constexpr int teams_of(int warps) { return PL::TEAM <= 32 ? warps * PL::TPW : warps / PL::WPT; }
  static constexpr int fit_warps(int w) {  // fewer where shared memory is short
    while (w > PL::WPT && team_bytes_x(1) * teams_of(w) + cta_bytes() > LIMIT) w -= PL::WPT;
    return w;
  }
  static constexpr int WARPS = fit_warps(REGS > 168 ? 8 : 4);
  static constexpr int TEAMS = teams_of(WARPS);
  // two exchange buffers (one barrier per exchange) when they fit, else one
  static constexpr int XBUF = team_bytes_x(2) * TEAMS + cta_bytes() <= LIMIT ? 2 : 1;
  static constexpr size_t team_bytes() { return team_bytes_x(XBUF); }
  static constexpr size_t smem() { return team_bytes() * TEAMS + cta_bytes(); }
};

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Compile-time loops whose index the bodies need as a constant.
template <int I, int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(static_cast<F&&>(f));
  }
}

template <class PL, bool SPLIT, int PH>
__global__ void __launch_bounds__(32 * FusedRegGeom<PL, SPLIT, PH>::WARPS, FusedRegGeom<PL, SPLIT, PH>::MINB)
    k_fused_reg(Dims d, const float2* __restrict__ tw, FusedArgs a, int nblk, int nteams) {
  typedef FusedRegGeom<PL, SPLIT, PH> G;
  typedef float2 C;
  constexpr int T = PL::T, A = PL::A, B = PL::B, K = PL::K, N = PL::N, W = PL::W, TEAM = PL::TEAM, SB = PL::SB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x;
  int team, tl;  // team within the CTA, lane within the team
  unsigned mask = 0xffffffffu;
  if constexpr (TEAM <= 32) {
    constexpr int used = PL::TPW * TEAM;
    if constexpr (used < 32) mask = (1u << used) - 1u;
    const int wt = lane / TEAM;
    team = warp * PL::TPW + wt;
    tl = lane - wt * TEAM;
  } else {
    team = warp / PL::WPT;
    tl = tid - team * TEAM;
  }
  // tables shared by the CTA: W_N^(j u) at [u][j] (row stride T + 1), longitude factors of the Coriolis term
  C* const stw = reinterpret_cast<C*>(smem_raw);
  float* const sct = reinterpret_cast<float*>(stw + K * (T + 1));
  for (int e = tid; e < K * T; e += nt) {
    const int u = e / T, j = e - u * T;
    stw[u * (T + 1) + j] = tw[(u * j) % N];
  }
  if constexpr (PH == FUSED_VELOCITY) {
    for (int e = tid; e < N; e += nt) sct[e] = (float)a.cth[e < d.nlat - 1 ? e : d.nlat - 1];
  }
  unsigned char* const mine = smem_raw + G::cta_bytes() + G::team_bytes() * team;
  float4* const sin_ = reinterpret_cast<float4*>(mine);
  C* const ex0 = reinterpret_cast<C*>(sin_ + G::STAGES * G::IN);
  C* const keep = ex0 + G::XBUF * G::EX;  // temperature phase: the velocity component in use, [K][TEAM]

  const int M = d.M;
  const int tot = (M + 1) * 2;
  const bool idle = TEAM <= 32 && lane >= PL::TPW * TEAM;  // lanes beyond the warp's teams
  if (!idle)
    for (int e = tl; e < G::STAGES * G::IN; e += TEAM) {
      const int w = e % G::IN;
      if (w >= tot) sin_[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  __syncthreads();
  if (idle) return;
  auto sync = [&] {
    if constexpr (TEAM <= 32) __syncwarp(mask);
    else asm volatile("bar.sync %0, %1;\n" ::"r"(team + 1), "n"(TEAM) : "memory");
  };
  const int j = tl >> 1, ii = tl & 1;

  // Outputs of this CTA: all of the phase, or blockIdx.y of two; they take the
  // components c0 .. c1 - 1 (a.fin: theta components, for the phi output 1, then phi components)
  const bool apart = PH != FUSED_TEMPERATURE && gridDim.y == 2;
  const int nin = PH == FUSED_INDUCTION ? 4 : a.nin, half = nin / 2;
  const int c0 = apart && blockIdx.y == 0 ? half : 0, c1 = apart && blockIdx.y == 1 ? half : nin;
  // input run of team index g and component c into stage st
  auto fetch = [&](int g, int c, int st) {
    const float4* src = a.fin[c] + (size_t)g * tot;
    float4* dst = sin_ + st * G::IN;
    for (int e = tl; e < tot; e += TEAM) cp_async16(dst + e, src + e);
    cp_async_commit();
  };
  // conjugated spectrum y_k (the inverse transform is conj(FFT(conj(Z)))) of
  // Z_k = F_N + i F_S and Z_(N-k) = conj(F_N) + i conj(F_S): k = j + T R
  const float4* const lo = sin_ + j * 2 + ii;          // order m = j + T R at lo + 2 T R
  const float4* const hi = sin_ + (T - j) * 2 + ii;    // order m = N - k = T - j + T (K - 1 - R)
  auto load_y = [&](auto Rc, int st) -> C {
    constexpr int R = decltype(Rc)::value;
    if constexpr (2 * R < K) {
      const float4 v = lo[st * G::IN + 2 * T * R];
      C y = make_float2(v.x - v.w, -(v.y + v.z));
      if constexpr (R == 0) {
        if (j == 0) y = make_float2(v.x, -v.z);
      }
      return y;
    } else {
      const float4 v = hi[st * G::IN + 2 * T * (K - 1 - R)];
      return make_float2(v.x + v.w, v.y - v.z);
    }
  };
  // sums of products, (north, -south) as the transforms deliver the grid rows
  C acc[K];
  int xb = 0;          // exchange buffer in use
  int st = 0;          // stage of the next component
  int gc = 0, gn = 0;  // team index in work and the next one (-1: none)
  C* const exr = ex0 + ii * PL::RO;

  // Inverse transform of the staged component c; consume(base index, A q + a, z[T])
  // gets the T longitudes phi = A q + a + K p of each (a, w) as (north, -south).
  auto inverse = [&](int c, auto&& consume) {
    cp_async_wait<0>();
    sync();
    [[maybe_unused]] C y[G::HOLD ? (SPLIT ? 2 * B : K) : 1];
    auto next = [&](int stage) {
      if (c + 1 < c1) fetch(gc, c + 1, stage);
      else if (gn >= 0) fetch(gn, c0, stage);
    };
    if constexpr (G::HOLD) {
      if constexpr (SPLIT) {
        static_for<0, B>([&](auto rr) {
          constexpr int R = decltype(rr)::value;
          y[R] = load_y(std::integral_constant<int, R>{}, 0);
          y[B + R] = load_y(std::integral_constant<int, R + 2 * B>{}, 0);
        });
      } else {
        static_for<0, K>([&](auto rr) { y[decltype(rr)::value] = load_y(rr, 0); });
      }
      sync();  // every lane has its part of the stage
      next(0);
      if constexpr (!SPLIT && A > 1) {
        static_for<0, B>([&](auto rr) {
          constexpr int R = decltype(rr)::value;
          C t[A];
#pragma unroll
          for (int s = 0; s < A; ++s) t[s] = y[R + B * s];
          RDft<A, C>::run(t);
          static_for<0, A>([&](auto aa) {
            constexpr int Q = decltype(aa)::value;
            y[R + B * Q] = mul_root<(long)R * Q, K>(t[Q]);
          });
        });
      }
    } else {
      next(st ^ 1);
    }
    static_for<0, A>([&](auto aa) {
      constexpr int Q = decltype(aa)::value;
      C v[B];
      static_for<0, B>([&](auto rr) {
        constexpr int R = decltype(rr)::value;
        if constexpr (SPLIT) {
          const C u = y[R], x = y[B + R];
          if constexpr (Q == 0) v[R] = cadd(u, x);
          else v[R] = mul_root<(long)R * Q, K>(cadd(u, mul_root<2 * Q, 3>(x)));
        } else if constexpr (G::HOLD) {
          v[R] = y[R + B * Q];
        } else {
          C s = load_y(std::integral_constant<int, R>{}, st);
          static_for<1, A>([&](auto ss) {
            constexpr int S = decltype(ss)::value;
            s = cadd(s, mul_root<(long)S * Q, A>(load_y(std::integral_constant<int, R + B * S>{}, st)));
          });
          v[R] = mul_root<(long)R * Q, K>(s);
        }
      });
      RDft<B, C>::run(v);
      C* const ex = exr + (G::XBUF == 2 ? xb * G::EX : 0);
      if constexpr (G::XBUF == 1) sync();  // the reads of the exchange before
#pragma unroll
      for (int q = 0; q < B; ++q) ex[j * SB + q] = cmul(v[q], stw[(A * q + Q) * (T + 1) + j]);
      sync();
#pragma unroll
      for (int w = 0; w < W; ++w) {
        C z[T];
#pragma unroll
        for (int p = 0; p < T; ++p) z[p] = ex[p * SB + j + T * w];
        RDft<T, C>::run(z);
        consume((Q * W + w) * T, A * (j + T * w) + Q, z);
      }
      xb ^= 1;
    });
    if constexpr (!G::HOLD) st ^= 1;
  };

  // Forward transform of acc and the folds w (G_N +- G_S) of product o.
  const float scl = (float)(0.5 * 2.0 * 3.14159265358979323846 / N);
  auto forward = [&](int o, int r, int ib, bool live) {
    constexpr int NZ = SPLIT ? 2 * B : K;
    C Z[NZ];
    static_for<0, A>([&](auto aa) {
      constexpr int Q = decltype(aa)::value;
      C* const ex = exr + (G::XBUF == 2 ? xb * G::EX : 0);
      if constexpr (G::XBUF == 1) sync();
#pragma unroll
      for (int w = 0; w < W; ++w) {
        C z[T];
#pragma unroll
        for (int p = 0; p < T; ++p) z[p] = acc[(Q * W + w) * T + p];
        RDft<T, C>::run(z);
        const int q = j + T * w;
        const C* const twq = stw + (A * q + Q) * (T + 1);
#pragma unroll
        for (int p = 0; p < T; ++p) ex[p * SB + q] = cmul(z[p], twq[p]);
      }
      sync();
      C v[B];
#pragma unroll
      for (int q = 0; q < B; ++q) v[q] = ex[j * SB + q];
      RDft<B, C>::run(v);
      if constexpr (SPLIT) {
        static_for<0, B>([&](auto rr) {
          constexpr int R = decltype(rr)::value;
          const C t = mul_root<(long)R * Q, K>(v[R]);
          if constexpr (Q == 0) {
            Z[R] = t;
            Z[B + R] = t;
          } else {
            Z[R] = cadd(Z[R], t);
            Z[B + R] = cadd(Z[B + R], mul_root<2 * Q, 3>(t));
          }
        });
      } else {
        static_for<0, B>([&](auto rr) {
          constexpr int R = decltype(rr)::value;
          Z[R + B * Q] = mul_root<(long)R * Q, K>(v[R]);
        });
      }
      xb ^= 1;
    });
    if constexpr (!SPLIT && A > 1) {
#pragma unroll
      for (int R = 0; R < B; ++R) {
        C t[A];
#pragma unroll
        for (int s = 0; s < A; ++s) t[s] = Z[R + B * s];
        RDft<A, C>::run(t);
#pragma unroll
        for (int s = 0; s < A; ++s) Z[R + B * s] = t[s];
      }
    }
    // Z at k = j + T R; the folds of order m need Z_m (thread j = m mod T) and
    // Z_(N-m), which thread T - j holds: the upper half goes through shared memory
    constexpr int NLO = SPLIT ? B : K / 2;
    C* const zx = ex0;  // orders 1 .. T NLO of both pairs
    static_assert(2 * (T * NLO + 1) <= G::EX, "mirror rows exceed the exchange buffer");
    sync();
#pragma unroll
    for (int R = 0; R < NLO; ++R) zx[(T - j + T * (NLO - 1 - R)) * 2 + ii] = Z[NLO + R];
    sync();
    const int ith = ib * 2 + ii;
    if (live && ith < d.nth) {
      const float h = scl * (float)a.w[ith];
      float2* const out = a.G + ((size_t)(o * d.nr + r) * (M + 1)) * 2 * d.nth + ith;
#pragma unroll
      for (int R = 0; R < NLO; ++R) {
        const int m = j + T * R;
        if (m > M) continue;
        const C zk = Z[R];
        C zn = zx[m * 2 + ii];
        if (R == 0 && j == 0) zn = zk;
        // with rows (N, -S): N_m = (Z_m + conj Z_(N-m)) / 2, S_m = i (Z_m - conj Z_(N-m)) / 2
        const float xx = zk.x + zn.x, xy = zk.y - zn.y, yx = -(zk.y + zn.y), yy = zk.x - zn.x;
        out[((size_t)m * 2 + 0) * d.nth] = make_float2(h * (xx + yx), h * (xy + yy));
        out[((size_t)m * 2 + 1) * d.nth] = make_float2(h * (xx - yx), h * (xy - yy));
      }
    }
    sync();  // the mirrored rows are read before the next exchange writes them
  };

  // The radial components are zero; every product with one is formed, as the
  // product of the other factor with (coefficient x 0).
  const float ur = 0.f, wr = 0.f, jr = 0.f, br = 0.f;
  // a warp's teams, and the warps of a team, run the same number of rounds;
  // a team past the last one repeats the last and stores nothing
  const int per_cta = G::teams_of(nt / 32), first = blockIdx.x * per_cta, stride = gridDim.x * per_cta;
  gn = min(first + team, nteams - 1);
  fetch(gn, c0, 0);
  for (int base = first; base < nteams; base += stride) {
    gc = gn;
    const bool live = base + team < nteams;
    gn = base + stride < nteams ? min(base + stride + team, nteams - 1) : -1;
    const int r = gc / nblk, ib = gc - r * nblk;
    if constexpr (PH == FUSED_TEMPERATURE) {
      // inputs g_r, u_th, g_th, u_ph, g_ph: -(u_r g_r + u_th g_th + u_ph g_ph) + S(r)
      const float s_r = (float)a.sources[r];
      C* const kp = keep + tl;
      for (int c = 0; c < 5; ++c) {
        inverse(c, [&](int e0, int, C* z) {
          if (c == 0) {
#pragma unroll
            for (int p = 0; p < T; ++p) acc[e0 + p] = make_float2(ur * z[p].x, ur * z[p].y);
          } else if (c & 1) {
#pragma unroll
            for (int p = 0; p < T; ++p) kp[(e0 + p) * TEAM] = make_float2(z[p].x, -z[p].y);
          } else {
#pragma unroll
            for (int p = 0; p < T; ++p) acc[e0 + p] = __ffma2_rn(kp[(e0 + p) * TEAM], z[p], acc[e0 + p]);
          }
        });
      }
#pragma unroll
      for (int e = 0; e < K; ++e) {
        float x = -acc[e].x, y = -acc[e].y;
        if (s_r != 0.f) { x += s_r; y -= s_r; }
        acc[e] = make_float2(x, y);
      }
      forward(0, r, ib, live);
    } else {
      // velocity: u, w, j, b (theta, phi each); the theta product from the phi components and the reverse:
      //   theta: adv (u_ph w_r - u_r w_ph) + mrf (-ct u_ph) + lf (j_ph b_r - j_r b_ph)
      //   phi:   adv (u_r w_th - u_th w_r) + mrf (ct u_th + st u_r) + lf (j_r b_th - j_th b_r)
      // induction: u, b: theta u_ph b_r - u_r b_ph, phi u_r b_th - u_th b_r
      const float rf_r = d.rfs32 ? d.rfs32[r] : a.rf;
      const float adv = -rf_r, mrf = a.cf != 0.f ? -rf_r : -a.cf, lfr = d.rfs32 ? rf_r : a.lf;
      for (int o = c0 == 0; o >= (c1 == half); --o) {
        const float sg = o ? -1.f : 1.f;  // sign of the first term of each product pair
#pragma unroll
        for (int e = 0; e < K; ++e) acc[e] = make_float2(0.f, 0.f);
        for (int c = 0; c < half; ++c) {
          float kz;
          if constexpr (PH == FUSED_INDUCTION) kz = c == 0 ? sg * br : -sg * ur;
          else kz = c == 0 ? adv * (sg * wr) : c == 1 ? adv * (-sg * ur) : c == 2 ? lfr * (sg * br) : lfr * (-sg * jr);
          const float2 kz2 = make_float2(kz, kz);
          const float kc = o ? mrf : -mrf;
          inverse(o ? c : half + c, [&](int e0, int ph0, C* z) {
#pragma unroll
            for (int p = 0; p < T; ++p) acc[e0 + p] = __ffma2_rn(kz2, z[p], acc[e0 + p]);
            if (PH == FUSED_VELOCITY && c == 0) {
#pragma unroll
              for (int p = 0; p < T; ++p) {
                const float f = kc * sct[ph0 + K * p];
                acc[e0 + p] = __ffma2_rn(make_float2(f, f), z[p], acc[e0 + p]);
              }
            }
          });
        }
        forward(o, r, ib, live);
      }
    }
  }
}

template <class PL, bool SPLIT, int PH>
void launch_fused_team(cudaStream_t s, const Dims& d, const float2* tw, const FusedArgs& a) {
  typedef FusedRegGeom<PL, SPLIT, PH> G;
  static_assert(G::smem() <= G::LIMIT, "shared memory");
  const int nblk = fourier_blocks(d), nteams = nblk * d.nr, sms = current_sm_count();
  // A handle with the chip to itself whose teams do not give every SM a full CTA: CTAs
  // of just enough warps, and each output to CTAs of its own while those fit the SMs
  // once (beyond, two rounds of one output take longer than one of both: lmax 47, nr
  // 260 velocity 33 against 31 us).  Packed into full CTAs a team took its outputs one
  // after the other on a few SMs (velocity / temperature / induction phase at lmax 127,
  // nlon 384, nr 9: 43 / 29 / 29 us, now 21 / 23 / 16; the passes of a whole CTA through
  // shared memory took 27 / 18 / 17).
  const bool spread = !a.dense && nteams < G::TEAMS * sms;
  const int outputs = spread && PH != FUSED_TEMPERATURE && 2 * nteams <= G::TEAMS * sms ? 2 : 1;
  int warps = spread ? PL::WPT : G::WARPS;
  while (warps < G::WARPS && G::teams_of(warps) * sms < nteams * outputs) warps += PL::WPT;
  const int teams = G::teams_of(warps), ctas = ceil_div(nteams, teams), most = sms * G::MINB;
  allow_dynamic_smem(k_fused_reg<PL, SPLIT, PH>, G::smem());
  k_fused_reg<PL, SPLIT, PH><<<dim3(ctas < most ? ctas : most, outputs), 32 * warps,
                               G::cta_bytes() + G::team_bytes() * teams, s>>>(d, tw, a, nblk, nteams);
}

template <class PL, bool SPLIT>
void launch_fused_plan(cudaStream_t s, const Dims& d, const float2* tw, int phase, const FusedArgs& a) {
  switch (phase) {
    case FUSED_TEMPERATURE: launch_fused_team<PL, SPLIT, FUSED_TEMPERATURE>(s, d, tw, a); break;
    case FUSED_VELOCITY: launch_fused_team<PL, SPLIT, FUSED_VELOCITY>(s, d, tw, a); break;
    default: launch_fused_team<PL, SPLIT, FUSED_INDUCTION>(s, d, tw, a); break;
  }
}

// Row length N = T A B; A = 3 also in its SPLIT form when the orders allow it.  Where
// the spectrum is not held (K > 40) a transform sums A points for each of A B values,
// so such a length takes the split with the smaller A: 360 as 6 5 12 against 6 10 6,
// velocity / temperature / induction phase at lmax 170, nr 33: 126 / 87 / 84 -> 84 / 60
// / 56 us, nr 5: 126 / 84 / 83 -> 49 / 58 / 35 (plan at run time: 56 / 38 / 35).
template <int T, int A, int B>
bool launch_fused_row(cudaStream_t s, const Dims& d, const void* twf, int phase, const FusedArgs& a) {
  typedef RowPlan<T, A, B> PL;
  const float2* tw = static_cast<const float2*>(twf);
  if constexpr (A == 3) {
    if (d.M < PL::N / 3) {
      launch_fused_plan<PL, true>(s, d, tw, phase, a);
      return true;
    }
  }
  launch_fused_plan<PL, false>(s, d, tw, phase, a);
  return true;
}

}  // namespace gd
