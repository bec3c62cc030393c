// gd_cnab2.cu -- the CNAB2 implicit step for every (field, l, m) radial system
// in one launch, energy diagnostics and a finite-value scan.
//
// build_rhs_cnab2! (src/timestep.jl:610-690):
//   rhs = u/dt + 1.5 N - 0.5 N_prev + (1 - theta) L_l u
// solve_implicit_step! + solve_banded! (src/timestep.jl:692-730,
// src/linear_algebra.jl:59-88): forward substitution with the unit lower
// factor, back substitution with the upper factor.  One thread owns one (l, m)
// column of one field and walks r with register windows; Re and Im share the
// factors.  The AB bootstrap (src/simulation.jl:1153-1170) is folded into the
// same pass; the history roll (:1312-1329) is the handle's switch of the two
// banks of nonlinear terms after the step (N_prev is read from the other bank).
#include "gd_internal.cuh"

namespace gd {

// The sweeps one at a time, for the host-array entry points (each runs some of
// them).  One thread solves the (l, m) column of one field, each sweep
// with loads that do not depend on the running recurrence so the unrolled
// loops keep many loads in flight:
//   1. rhs = u/dt + 1.5 N - 0.5 N_prev + (1 - theta) L_l u  (written over u);
//   2. forward substitution with the unit lower factor (y over u);
//   3. back substitution with the upper factor (x over u).
// L_l = nu lap - nu l(l+1)/r^2 is rebuilt from the block's shared Laplacian
// band with the same roundings as the set-up kernel.
template <int KL>
__device__ __forceinline__ void cnab2_column(const Dims& d, int j, int l, const double* __restrict__ LU,
                                             const double* __restrict__ sband, const double* __restrict__ srinv2,
                                             double nu, const Cnab2Args& a, int slot, int N, int base) {
  // the segment's N levels start at shell base; the planes span all shells
  const size_t NM = d.nlm, plane = (size_t)d.nr * NM;
  const size_t Lp1 = (size_t)d.L + 1;
  constexpr int NB = 2 * KL + 1;
  const double nulf = __dmul_rn(nu, (double)l * (l + 1));
  const size_t s0 = (size_t)base * NM + j;
  double* __restrict__ ure = a.u[slot] + s0;
  double* __restrict__ uim = a.u[slot] + plane + s0;
  const double* __restrict__ nre = a.nl[slot] + s0;
  const double* __restrict__ nim = a.nl[slot] + plane + s0;
  const double* __restrict__ pre = a.prev[slot] + s0;
  const double* __restrict__ pim = a.prev[slot] + plane + s0;
  const double* __restrict__ F = LU + l;
  const bool boot = a.boot != 0;
  const bool rows = a.bc_rows != 0;
  const double* __restrict__ rowv = a.rowvals[slot];
  const int stages = a.stages ? a.stages : 7;

  // sweep 1: right-hand side, rows in batches of RB whose loads are issued first
  constexpr int RB = 4;
  if (stages & 1) {
    double wr[NB], wi[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const int idx = t - KL;
      wr[t] = (idx >= 0 && idx < N) ? ure[(size_t)idx * NM] : 0.0;
      wi[t] = (idx >= 0 && idx < N) ? uim[(size_t)idx * NM] : 0.0;
    }
    for (int i0 = 0; i0 < N; i0 += RB) {
      double unr[RB], uni[RB], nr_[RB], ni_[RB], pr_[RB], pi_[RB];
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const int i = i0 + b, nxt = i + KL + 1;
        unr[b] = (nxt < N) ? ure[(size_t)nxt * NM] : 0.0;
        uni[b] = (nxt < N) ? uim[(size_t)nxt * NM] : 0.0;
        if (i < N) {
          nr_[b] = nre[(size_t)i * NM];
          ni_[b] = nim[(size_t)i * NM];
          pr_[b] = boot ? nr_[b] : pre[(size_t)i * NM];
          pi_[b] = boot ? ni_[b] : pim[(size_t)i * NM];
        } else {
          nr_[b] = ni_[b] = pr_[b] = pi_[b] = 0.0;
        }
      }
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const int i = i0 + b;
        if (i >= N) break;
        const size_t at = (size_t)i * NM;
        double Lr = 0.0, Li = 0.0;
#pragma unroll
        for (int t = 0; t < NB; ++t) {
          const int col = i - KL + t;
          if (col >= 0 && col < N) {
            double cf = sband[col * NB + (KL + i - col)];
            if (t == KL) cf = __dsub_rn(cf, __dmul_rn(nulf, srinv2[i]));
            Lr += cf * wr[t];
            Li += cf * wi[t];
          }
        }
        double vr = a.inv_dt * wr[KL] + 1.5 * nr_[b] - 0.5 * pr_[b];
        double vi = a.inv_dt * wi[KL] + 1.5 * ni_[b] - 0.5 * pi_[b];
        vr += a.lin_weight * Lr;
        vi += a.lin_weight * Li;
        if (rows && (i == 0 || i == N - 1)) {
          // ball: the r = 0 row of l >= 1 is the regularity condition (value 0)
          vr = (rowv != nullptr && !(d.ball && i == 0 && l > 0)) ? rowv[(i == 0 ? 0 : NM) + j] : 0.0;
          vi = 0.0;
        }
        ure[at] = vr;
        uim[at] = vi;
#pragma unroll
        for (int t = 0; t < NB - 1; ++t) { wr[t] = wr[t + 1]; wi[t] = wi[t + 1]; }
        wr[NB - 1] = unr[b];
        wi[NB - 1] = uni[b];
      }
    }
  }
  // sweep 2: forward substitution (unit lower factor), y[i - KL + t] in yr[t]
  if (stages & 2) {
  double yr[KL], yi[KL];
#pragma unroll
  for (int t = 0; t < KL; ++t) yr[t] = yi[t] = 0.0;
  for (int i0 = 0; i0 < N; i0 += RB) {
    double br[RB], bi[RB], lf[RB][KL];
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = i0 + b;
      br[b] = (i < N) ? ure[(size_t)i * NM] : 0.0;
      bi[b] = (i < N) ? uim[(size_t)i * NM] : 0.0;
#pragma unroll
      for (int t = 0; t < KL; ++t) {
        const int col = i - KL + t;
        lf[b][t] = (i < N && col >= 0) ? F[((size_t)col * NB + (KL + i - col)) * Lp1] : 0.0;
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = i0 + b;
      if (i >= N) break;
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int t = 0; t < KL; ++t) {
        if (i - KL + t >= 0) {
          sr += lf[b][t] * yr[t];
          si += lf[b][t] * yi[t];
        }
      }
      const double y_r = br[b] - sr, y_i = bi[b] - si;
      ure[(size_t)i * NM] = y_r;
      uim[(size_t)i * NM] = y_i;
#pragma unroll
      for (int t = 0; t < KL - 1; ++t) { yr[t] = yr[t + 1]; yi[t] = yi[t + 1]; }
      yr[KL - 1] = y_r;
      yi[KL - 1] = y_i;
    }
  }
  }
  // sweep 3: back substitution, x[i + 1 + t] in xr[t]
  if (stages & 4) {
  double xr[KL], xi[KL];
#pragma unroll
  for (int t = 0; t < KL; ++t) xr[t] = xi[t] = 0.0;
  for (int i0 = N - 1; i0 >= 0; i0 -= RB) {
    double yv[RB], yw[RB], uf[RB][KL], dg[RB];
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = i0 - b;
      yv[b] = (i >= 0) ? ure[(size_t)i * NM] : 0.0;
      yw[b] = (i >= 0) ? uim[(size_t)i * NM] : 0.0;
      dg[b] = (i >= 0) ? F[((size_t)i * NB + KL) * Lp1] : 1.0;
#pragma unroll
      for (int t = 0; t < KL; ++t) {
        const int col = i + 1 + t;
        uf[b][t] = (i >= 0 && col < N) ? F[((size_t)col * NB + (KL + i - col)) * Lp1] : 0.0;
      }
    }
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      const int i = i0 - b;
      if (i < 0) break;
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int t = 0; t < KL; ++t) {
        if (i + 1 + t < N) {
          sr += uf[b][t] * xr[t];
          si += uf[b][t] * xi[t];
        }
      }
      const double x_r = (yv[b] - sr) / dg[b];
      const double x_i = (yw[b] - si) / dg[b];
      // bc_mode 1 zeroes the boundary rows after the whole solve: the
      // substitution itself continues with the solved values
      const bool clamp = a.clamp_rows && (i == 0 || i == N - 1);
      ure[(size_t)i * NM] = clamp ? 0.0 : x_r;
      uim[(size_t)i * NM] = clamp ? 0.0 : x_i;
#pragma unroll
      for (int t = KL - 1; t > 0; --t) { xr[t] = xr[t - 1]; xi[t] = xi[t - 1]; }
      xr[0] = x_r;
      xi[0] = x_i;
    }
  }
  }
}

// blockIdx.y = field slot; the block's Laplacian band uses that field's diffusivity.
template <int KL>
// 160 registers, three 128-thread blocks per SM (more columns in flight than
// wider row batches would give)
__global__ void __launch_bounds__(128, 3) k_cnab2(Dims d, const int* __restrict__ lof, const double* __restrict__ d1,
                                               const double* __restrict__ d2, const double* __restrict__ rinv,
                                               const double* __restrict__ rinv2, const double* __restrict__ nu,
                                               const double* __restrict__ lu, Cnab2Args a) {
  constexpr int NB = 2 * KL + 1;
  extern __shared__ double sm[];
  double* sband = sm;                 // nu * lap, [col][band]
  double* srinv2 = sm + (size_t)d.nrs * NB;
  const int slot = blockIdx.y;
  if (slot >= a.nfield) return;
  const int g = a.kind[slot];
  const double nuk = nu[g];
  // the segment's radial operators (its variant's band, its shells' 1/r)
  const SegView sv = seg_view(d, blockIdx.z);
  const int N = sv.n;
  d1 += sv.band_off;
  d2 += sv.band_off;
  rinv += sv.base;
  rinv2 += sv.base;
  lu += sv.op_off;
  for (int e = threadIdx.x; e < N * NB; e += blockDim.x) {
    const int col = e / NB, b = e % NB, i = col + b - KL;
    double v = 0.0;
    if (i >= 0 && i < N) {
      const size_t q = b + (size_t)NB * col;
      // same roundings as the set-up kernel: nu * (d2 + (2 r^-1) d1)
      v = __dmul_rn(nuk, __dadd_rn(d2[q], __dmul_rn(__dmul_rn(2.0, rinv[i]), d1[q])));
    }
    sband[e] = v;
  }
  for (int i = threadIdx.x; i < N; i += blockDim.x) srinv2[i] = rinv2[i];
  __syncthreads();
  const int j = d.jlo + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.jhi) return;
  const int l = lof[j];
  const double* LUk = lu + (size_t)g * N * NB * ((size_t)d.L + 1);
  const int* rt = a.rowtypes[slot];
  if (a.bc_rows && rt != nullptr && a.lu_flux != nullptr) {
    // a prescribed flux at a boundary: the factors with the row of D1 there
    const int fv = (rt[j] == GD_BC_FLUX ? 1 : 0) | (rt[d.nlm + j] == GD_BC_FLUX ? 2 : 0);
    if (fv)
      LUk = a.lu_flux + (size_t)(fv - 1) * a.lu_flux_stride + sv.op_off + (size_t)g * N * NB * ((size_t)d.L + 1);
  }
  cnab2_column<KL>(d, j, l, LUk, sband, srinv2, nuk, a, slot, N, sv.base);
}

// ---------------------------------------------------------------------------
// The whole step of a column.
//
// Packed operators (launch_pack_lu), rows i of kind g, l fastest: double2
//   fac [g][i][5][l]: (L_-4, L_-3), (L_-2, L_-1), (1 / U_0, U_0), (U_1, U_2), (U_3, U_4)
// of the factors' row i (zero outside the matrix), and doubles
//   row [g][i][10]: the nine coefficients of nu lap at columns i - 4 .. i + 4, then r^-2.
// Upward pass: right-hand side and forward substitution (the window keeps the
// original u the band needs, y is written over u); downward pass: back
// substitution.  Rows come in batches whose loads are issued one batch ahead.
//
// What bounds it: load latency (a row of a column is 64 bytes of fields and 80
// of factors, and its substitution waits for the row before).  The single sweeps
// above execute about 470 warp instructions a row (ncu, 79.4 M for 5 x 32896
// columns of 33 rows): they shift their windows, test every column, form 64-bit
// factor offsets and divide.  Here nine rows are unrolled per round, so a window
// index is a constant; factors come as 16-byte loads at 32-bit offsets from
// uniform bases; no column is tested (tables and windows are zero outside the
// matrix); the stored reciprocal with one correction step (quotient()) stands for
// the division.  The terms are read once, past the caches' retention, so that y
// still lies in L2 when the downward pass reads it; two blocks of 128 threads
// with a batch of loads in flight beat three without one where the columns fill
// the chip unevenly.  Measured (B200, six-field or five-field step, before ->
// after): lmax 255, nr 129: 576 -> 438 us; lmax 341, nr 33: 276 -> 197; lmax 140,
// nr 97: 244 -> 138; lmax 127, nr 65: 106 -> 83; lmax 31, nr 32: 43 -> 21 us.
// Four blocks of 128 registers ran at 642 us (y falls out of L2); both potentials
// of a vector in one block, sharing factor loads, gained under 1%.
// ---------------------------------------------------------------------------
__global__ void k_pack_lu(int N, int Lp1, const double* __restrict__ d1, const double* __restrict__ d2,
                          const double* __restrict__ rinv, const double* __restrict__ rinv2,
                          const double* __restrict__ nu, const double* __restrict__ lu, double2* __restrict__ fac,
                          double* __restrict__ row) {
  constexpr int KL = GD_MAX_KL, NB = GD_NBW;
  const int i = blockIdx.x, g = blockIdx.y;
  for (int l = threadIdx.x; l < Lp1; l += blockDim.x) {
    auto at = [&](int col) {
      return (col >= 0 && col < N) ? lu[(((size_t)g * N + col) * NB + (KL + i - col)) * Lp1 + l] : 0.0;
    };
    double2* o = fac + ((size_t)(g * N + i) * 5) * Lp1 + l;
    o[0] = make_double2(at(i - 4), at(i - 3));
    o[(size_t)Lp1] = make_double2(at(i - 2), at(i - 1));
    o[(size_t)2 * Lp1] = make_double2(__drcp_rn(at(i)), at(i));
    o[(size_t)3 * Lp1] = make_double2(at(i + 1), at(i + 2));
    o[(size_t)4 * Lp1] = make_double2(at(i + 3), at(i + 4));
  }
  if (row != nullptr && threadIdx.x < NB + 1) {
    const int t = threadIdx.x, col = i - KL + t;
    double v = 0.0;
    if (t == NB) v = rinv2[i];
    else if (col >= 0 && col < N) {
      const size_t q = (KL + i - col) + (size_t)NB * col;
      // same roundings as the set-up kernel: nu * (d2 + (2 r^-1) d1)
      v = __dmul_rn(nu[g], __dadd_rn(d2[q], __dmul_rn(__dmul_rn(2.0, rinv[i]), d1[q])));
    }
    row[(size_t)(g * N + i) * (NB + 1) + t] = v;
  }
}

void launch_pack_lu(cudaStream_t s, int N, int L, int nkind, const double* d1, const double* d2, const double* rinv,
                    const double* rinv2, const double* nu, const double* lu, double2* fac, double* row) {
  k_pack_lu<<<dim3(N, nkind), 128, 0, s>>>(N, L + 1, d1, d2, rinv, rinv2, nu, lu, fac, row);
}

__device__ __forceinline__ double ldd(const char* p, unsigned off) { return *reinterpret_cast<const double*>(p + off); }
__device__ __forceinline__ double ldcs(const char* p, unsigned off) {
  return __ldcs(reinterpret_cast<const double*>(p + off));
}
__device__ __forceinline__ double2 ldf(const char* p, unsigned off) {
  return __ldg(reinterpret_cast<const double2*>(p + off));
}

__global__ void __launch_bounds__(128, 2) k_cnab2_step(Dims d, const int* __restrict__ lof, Cnab2Args a) {
  constexpr int KL = GD_MAX_KL, NB = GD_NBW, RW = NB + 1;
  static_assert(KL == 4, "the factor rows are packed for four off-diagonals");
  extern __shared__ __align__(16) double sm[];  // [N][RW]
  const int slot = blockIdx.y, g = a.kind[slot];
  const SegView sv = seg_view(d, blockIdx.z);
  const int N = sv.n;
  const unsigned Lp1 = d.L + 1;
  {
    const long oprow = sv.op_off / ((long)NB * Lp1);  // operator rows before this variant's
    const double* src = a.row + (oprow + (long)g * N) * RW;
    for (int e = threadIdx.x; e < N * RW; e += blockDim.x) sm[e] = src[e];
  }
  __syncthreads();
  const int j = d.jlo + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= d.jhi) return;
  const int l = lof[j];
  const unsigned NM8 = (unsigned)d.nlm * 8u;
  const size_t plane = (size_t)d.nr * d.nlm * 8;
  char* const ur = reinterpret_cast<char*>(a.u[slot]) + (size_t)sv.base * NM8;
  char* const ui = ur + plane;
  const char* const nr = reinterpret_cast<const char*>(a.nl[slot]) + (size_t)sv.base * NM8;
  const char* const ni = nr + plane;
  // an AB1 start takes the current terms for the previous ones
  const char* const pr = a.boot ? nr : reinterpret_cast<const char*>(a.prev[slot]) + (size_t)sv.base * NM8;
  const char* const pi = pr + plane;
  const char* const fac = reinterpret_cast<const char*>(a.fac);
  const unsigned fs = Lp1 * 16u;  // bytes between the factor pairs of a row
  unsigned f0 = (unsigned)(sv.op_off / NB) * 5u * 16u + (unsigned)g * N * 5u * fs + (unsigned)l * 16u;
  const int* rt = a.rowtypes[slot];
  if (a.bc_rows && rt != nullptr && a.fac_flux_stride != 0) {
    // a prescribed flux at a boundary: the factors with the row of D1 there
    const unsigned fv = (rt[j] == GD_BC_FLUX ? 1u : 0u) | (rt[d.nlm + j] == GD_BC_FLUX ? 2u : 0u);
    f0 += fv * (unsigned)(a.fac_flux_stride * 16);
  }
  const double nulf = __dmul_rn(a.nu[g], (double)l * (l + 1));
  const double* rowv = a.rowvals[slot];
  const double inv_dt = a.inv_dt, lw = a.lin_weight;
  const unsigned j8 = (unsigned)j * 8u;

  {
    constexpr int RB = 3;
    struct In { double nr, ni, pr, pi, ur, ui; double2 l0, l1; };
    In cur[RB], nxt[RB];
    auto load = [&](In* v, int i0) {
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const int i = i0 + b;
        if (i < N) {
          const unsigned o = j8 + (unsigned)i * NM8;
          v[b].nr = ldcs(nr, o); v[b].ni = ldcs(ni, o);
          v[b].pr = ldcs(pr, o); v[b].pi = ldcs(pi, o);
          const unsigned f = f0 + (unsigned)i * 5u * fs;
          v[b].l0 = ldf(fac, f); v[b].l1 = ldf(fac, f + fs);
        }
        v[b].ur = v[b].ui = 0.0;
        if (i + KL + 1 < N) {
          const unsigned o = j8 + (unsigned)(i + KL + 1) * NM8;
          v[b].ur = ldd(ur, o); v[b].ui = ldd(ui, o);
        }
      }
    };
    // u at rows i - 4 .. i + 4 of row i = i0 + b in slots (b .. b + 8) mod 9 (i0 a multiple of 9)
    double wr[NB], wi[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const int i = t - KL;
      wr[t] = wi[t] = 0.0;
      if (i >= 0 && i < N) { wr[t] = ldd(ur, j8 + (unsigned)i * NM8); wi[t] = ldd(ui, j8 + (unsigned)i * NM8); }
    }
    double yr[KL] = {0.0, 0.0, 0.0, 0.0}, yi[KL] = {0.0, 0.0, 0.0, 0.0};
    load(cur, 0);
    for (int i0 = 0; i0 < N; i0 += NB) {
#pragma unroll
      for (int sb = 0; sb < NB / RB; ++sb) {
        load(nxt, i0 + RB * (sb + 1));
#pragma unroll
        for (int bb = 0; bb < RB; ++bb) {
          const int b = RB * sb + bb, i = i0 + b;
          if (i < N) {
            const double* cf = sm + i * RW;
            double Lr = 0.0, Li = 0.0;
#pragma unroll
            for (int t = 0; t < NB; ++t) {
              double c = cf[t];
              if (t == KL) c = __dsub_rn(c, __dmul_rn(nulf, cf[NB]));
              Lr += c * wr[(b + t) % NB];
              Li += c * wi[(b + t) % NB];
            }
            const In& v = cur[bb];
            double vr = inv_dt * wr[(b + KL) % NB] + 1.5 * v.nr - 0.5 * v.pr;
            double vi = inv_dt * wi[(b + KL) % NB] + 1.5 * v.ni - 0.5 * v.pi;
            vr += lw * Lr;
            vi += lw * Li;
            if (a.bc_rows && (i == 0 || i == N - 1)) {
              // ball: the r = 0 row of l >= 1 is the regularity condition (value 0)
              vr = (rowv != nullptr && !(d.ball && i == 0 && l > 0)) ? rowv[(i == 0 ? 0 : d.nlm) + j] : 0.0;
              vi = 0.0;
            }
            const double sr = v.l0.x * yr[0] + v.l0.y * yr[1] + v.l1.x * yr[2] + v.l1.y * yr[3];
            const double si = v.l0.x * yi[0] + v.l0.y * yi[1] + v.l1.x * yi[2] + v.l1.y * yi[3];
            vr = vr - sr;
            vi = vi - si;
#pragma unroll
            for (int t = 0; t < KL - 1; ++t) { yr[t] = yr[t + 1]; yi[t] = yi[t + 1]; }
            yr[KL - 1] = vr;
            yi[KL - 1] = vi;
            const unsigned o = j8 + (unsigned)i * NM8;
            *reinterpret_cast<double*>(ur + o) = vr;
            *reinterpret_cast<double*>(ui + o) = vi;
          }
          wr[b] = cur[bb].ur;
          wi[b] = cur[bb].ui;
        }
#pragma unroll
        for (int bb = 0; bb < RB; ++bb) cur[bb] = nxt[bb];
      }
    }
  }
  {
    constexpr int RB = 4;
    struct In { double yr, yi; double2 dg, u0, u1; };
    In cur[RB], nxt[RB];
    auto load = [&](In* v, int i0) {  // rows i0, i0 - 1, ..
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const int i = i0 - b;
        if (i >= 0) {
          const unsigned o = j8 + (unsigned)i * NM8;
          v[b].yr = ldcs(ur, o); v[b].yi = ldcs(ui, o);
          const unsigned f = f0 + ((unsigned)i * 5u + 2u) * fs;
          v[b].dg = ldf(fac, f); v[b].u0 = ldf(fac, f + fs); v[b].u1 = ldf(fac, f + 2 * fs);
        }
      }
    };
    double xr[KL] = {0.0, 0.0, 0.0, 0.0}, xi[KL] = {0.0, 0.0, 0.0, 0.0};
    load(cur, N - 1);
    for (int i0 = N - 1; i0 >= 0; i0 -= RB) {
      load(nxt, i0 - RB);
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const int i = i0 - b;
        if (i >= 0) {
          const In& v = cur[b];
          const double tr = v.yr - (v.u0.x * xr[0] + v.u0.y * xr[1] + v.u1.x * xr[2] + v.u1.y * xr[3]);
          const double ti = v.yi - (v.u0.x * xi[0] + v.u0.y * xi[1] + v.u1.x * xi[2] + v.u1.y * xi[3]);
          const double x_r = quotient(tr, v.dg.y, v.dg.x), x_i = quotient(ti, v.dg.y, v.dg.x);
          // bc_mode 1 zeroes the boundary rows after the whole solve: the
          // substitution itself continues with the solved values
          const bool clamp = a.clamp_rows && (i == 0 || i == N - 1);
          const unsigned o = j8 + (unsigned)i * NM8;
          __stcs(reinterpret_cast<double*>(ur + o), clamp ? 0.0 : x_r);
          __stcs(reinterpret_cast<double*>(ui + o), clamp ? 0.0 : x_i);
#pragma unroll
          for (int t = KL - 1; t > 0; --t) { xr[t] = xr[t - 1]; xi[t] = xi[t - 1]; }
          xr[0] = x_r;
          xi[0] = x_i;
        }
      }
#pragma unroll
      for (int b = 0; b < RB; ++b) cur[b] = nxt[b];
    }
  }
}

void launch_cnab2(cudaStream_t s, const Dims& d, const int* lof, const double* d1, const double* d2,
                  const double* rinv, const double* rinv2, const double* nu, const double* lu, const Cnab2Args& a) {
  // (offsets of the whole-step kernel are 32-bit)
  const size_t top = (size_t)1 << 32;
  if (a.fac != nullptr && a.stages == 0 && a.fac_bytes < top && (size_t)d.nr * d.nlm * sizeof(double) < top) {
    // blocks small enough that a small model's columns reach every SM
    const int cols = d.jhi - d.jlo;
    int bs = 128;
    while (bs > 32 && (long)ceil_div(cols, bs) * a.nfield * d.nseg < 2L * current_sm_count()) bs /= 2;
    dim3 grid(ceil_div(cols, bs), a.nfield, d.nseg);
    const size_t smem = (size_t)d.nrs * (GD_NBW + 1) * sizeof(double);
    allow_dynamic_smem(k_cnab2_step, smem);
    Cnab2Args b = a;
    b.nu = nu;
    k_cnab2_step<<<grid, bs, smem, s>>>(d, lof, b);
    return;
  }
  dim3 grid(ceil_div(d.jhi - d.jlo, 128), a.nfield, d.nseg);
  const size_t smem = ((size_t)d.nrs * GD_NBW + d.nrs) * sizeof(double);
  k_cnab2<GD_MAX_KL><<<grid, 128, smem, s>>>(d, lof, d1, d2, rinv, rinv2, nu, lu, a);
}

// 0.5 sum over (r, l, m) of (T^2 + P^2) / max(l(l+1), 1) for velocity and
// magnetic fields (src/magnetic.jl:519-542).  Deterministic two-level sum,
// one per segment (blockIdx.y), each in the order of an unsegmented handle.
__global__ void k_energy_partial(Dims d, const int* __restrict__ lof, const double* __restrict__ ut,
                                 const double* __restrict__ up, const double* __restrict__ bt,
                                 const double* __restrict__ bp, double* __restrict__ partial) {
  __shared__ double sk[256], sm[256];
  const size_t NM = d.nlm, plane = (size_t)d.nr * NM;
  const SegView sv = seg_view(d, blockIdx.y);
  const size_t seg0 = (size_t)sv.base * NM, segn = (size_t)sv.n * NM;
  ut += seg0;
  up += seg0;
  if (bt) {
    bt += seg0;
    bp += seg0;
  }
  double ek = 0.0, em = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < segn; i += (size_t)gridDim.x * blockDim.x) {
    const int l = lof[i % NM];
    const double lfv = (double)l * (l + 1.0);
    const double w = 1.0 / (lfv > 1.0 ? lfv : 1.0);
    ek += w * (ut[i] * ut[i] + ut[plane + i] * ut[plane + i] + up[i] * up[i] + up[plane + i] * up[plane + i]);
    if (bt) em += w * (bt[i] * bt[i] + bt[plane + i] * bt[plane + i] + bp[i] * bp[i] + bp[plane + i] * bp[plane + i]);
  }
  sk[threadIdx.x] = ek;
  sm[threadIdx.x] = em;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) { sk[threadIdx.x] += sk[threadIdx.x + s]; sm[threadIdx.x] += sm[threadIdx.x + s]; }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const size_t q = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
    partial[2 * q] = sk[0];
    partial[2 * q + 1] = sm[0];
  }
}

// out[2 g], out[2 g + 1]: kinetic and magnetic energy of segment g
__global__ void k_energy_final(int nblk, int nseg, const double* __restrict__ partial, double* __restrict__ out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nseg) return;
  partial += (size_t)2 * nblk * g;
  double ek = 0.0, em = 0.0;
  for (int b = 0; b < nblk; ++b) { ek += partial[2 * b]; em += partial[2 * b + 1]; }
  out[2 * g] = 0.5 * ek;
  out[2 * g + 1] = 0.5 * em;
}

void launch_energy(cudaStream_t s, const Dims& d, const int* lof, const double* utor, const double* upol,
                   const double* btor, const double* bpol, double* partial, double* out) {
  const int nblk = GD_ENERGY_BLOCKS;
  k_energy_partial<<<dim3(nblk, d.nseg), 256, 0, s>>>(d, lof, utor, upol, btor, bpol, partial);
  k_energy_final<<<ceil_div(d.nseg, 32), 32, 0, s>>>(nblk, d.nseg, partial, out);
}

__global__ void k_check_finite(size_t n, const double* __restrict__ a, int* flag) {
  int bad = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (!isfinite(a[i])) bad = 1;
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(flag, 1);
}

void launch_check_finite(cudaStream_t s, size_t n, const double* a, int* flag) {
  k_check_finite<<<296, 256, 0, s>>>(n, a, flag);
}

}  // namespace gd
