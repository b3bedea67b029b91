// nbg_orbit.cuh -- the orbit producer: one GPU lane advances one system.
//
// Per AHL21 step (src/integrator/ahl21/ahl21.jl:5-95) the producer updates x,
// v (with their Kahan errors) and, when asked, dq/dt, exactly as the
// reference does, and emits the step's linear operators for the Jacobian
// consumer instead of applying them to jac_step itself:
//   * each Kepler pair (i, j): the 6x6 block K of jac_kepler, m_i/(m_i+m_j),
//     m_j/(m_i+m_j) and two 6-vectors that make up the two mass columns of
//     jac_ij (50 doubles) -- the 14x14 jac_ij of ahl21.jl:734-750 is exactly
//     these numbers (see PREC in nbg_layout.cuh);
//   * phic!/phisalpha! (ahl21.jl:392-700): jac_phi restricted to its only
//     non-zero block, velocity rows x (position, mass) columns (3N x 4N);
//   * kickfast! (ahl21.jl:337-386) for pair[i,j] == true: jac_kick on the
//     same block.
// The operators depend on x, v only, never on jac_step, so orbit and Jacobian
// are decoupled (the producer/consumer split of this package).
//
// Compact operator layout: row 3b + k is body b's velocity component k,
// column 4d + p is body d's position component p (p < 3) or mass (p == 3).
#pragma once
#include "../../include/nbg.h"
#include "nbg_layout.cuh"
#include "nbg_kepler.cuh"

namespace nbg {

// Record writer: element e of this lane's record at p[e * stride].
struct Rec {
  double* p;
  int stride;
  __device__ __forceinline__ void put(int e, double v) const {
    if (p) p[(size_t)e * stride] = v;
  }
  __device__ __forceinline__ double get(int e) const { return p[(size_t)e * stride]; }
};

template <int N>
struct Sys {
  double x[3 * N], v[3 * N], xe[3 * N], ve[3 * N], m[N];
  double dqdt[7 * N];
};

// x and v all finite (the State check of Integrator.jl:137-143, which the
// reference only prints; here it raises NBG_STATUS_NONFINITE).
template <int N>
__device__ __forceinline__ bool state_finite(const Sys<N>& st) {
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 3 * N; q++) ok = ok && isfinite(st.x[q]) && isfinite(st.v[q]);
  return ok;
}

// Scratch of one step (the Derivatives fields the producer needs,
// src/PreAllocArrays.jl:65-113), compact layouts.
template <int N>
struct Work {
  double op[12 * N * N];    // jac_kick or jac_phi block
  double dadq[12 * N * N];  // d a / d (x, m), rows 3i+k, cols 4d+p
  double dot[4 * N];
  double a[3 * N];
  double dqop[3 * N];       // dqdt_kick or dqdt_phi velocity entries
  // last pair's jac_ij (factored) and dqdt_ij: stale values are reused when
  // G (m_i + m_j) == 0, as ahl21.jl:713 returns before refilling them.
  double lk[36], lmi, lmj, lpsi[6], lb[6], ldq[14];
};

#define OPX(r, c) w.op[(r) * (4 * N) + (c)]
#define DAX(r, c) w.dadq[(r) * (4 * N) + (c)]

template <int N>
__device__ __forceinline__ void reset_last(Work<N>& w) {
  for (int q = 0; q < 36; q++) w.lk[q] = 0.0;
  w.lmi = w.lmj = 0.0;
  for (int q = 0; q < 6; q++) w.lpsi[q] = w.lb[q] = 0.0;
  for (int q = 0; q < 14; q++) w.ldq[q] = 0.0;
}

// drift (ahl21.jl:318-331 for x; the jac_step part is the consumer's)
template <int N>
__device__ __forceinline__ void drift(Sys<N>& s, double h) {
#pragma unroll
  for (int q = 0; q < 3 * N; q++) kahan(s.x[q], s.xe[q], h * s.v[q]);
}

// kickfast! (ahl21.jl:337-386 / ahl21_no_grad.jl:35-56)
template <int N>
__device__ void kickfast(Sys<N>& s, Work<N>& w, double h, uint64_t kick) {
  for (int q = 0; q < 12 * N * N; q++) w.op[q] = 0.0;
  for (int q = 0; q < 3 * N; q++) w.dqop[q] = 0.0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (!((kick >> pair_bit(i, j, N)) & 1)) continue;
      double rij[3];
      for (int k = 0; k < 3; k++) rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      double r2inv = 1.0 / (rij[0] * rij[0] + rij[1] * rij[1] + rij[2] * rij[2]);
      double r3inv = r2inv * sqrt(r2inv);
      double fac2 = h * GNEWT * r3inv;
      for (int k = 0; k < 3; k++) {
        double fac = fac2 * rij[k];
        kahan(s.v[3 * i + k], s.ve[3 * i + k], (-s.m[j]) * fac);
        kahan(s.v[3 * j + k], s.ve[3 * j + k], s.m[i] * fac);
        w.dqop[3 * i + k] = w.dqop[3 * i + k] - s.m[j] * fac / h;
        w.dqop[3 * j + k] = w.dqop[3 * j + k] + s.m[i] * fac / h;
        OPX(3 * i + k, 4 * j + 3) -= fac;
        OPX(3 * j + k, 4 * i + 3) += fac;
        fac = fac * (3.0 * r2inv);
        for (int p = 0; p < 3; p++) {
          OPX(3 * i + k, 4 * i + p) += fac * s.m[j] * rij[p];
          OPX(3 * i + k, 4 * j + p) -= fac * s.m[j] * rij[p];
          OPX(3 * j + k, 4 * j + p) += fac * s.m[i] * rij[p];
          OPX(3 * j + k, 4 * i + p) -= fac * s.m[i] * rij[p];
        }
        OPX(3 * i + k, 4 * i + k) -= fac2 * s.m[j];
        OPX(3 * i + k, 4 * j + k) += fac2 * s.m[j];
        OPX(3 * j + k, 4 * j + k) -= fac2 * s.m[i];
        OPX(3 * j + k, 4 * i + k) += fac2 * s.m[i];
      }
    }
}

// dqdt += dqop/div + op * dqdt (ahl21.jl:11-14, :51-52, :86-89); the gemv
// is one FMA chain per row in the reference's column order; columns with a
// zero operator entry or a zero dq/dt entry (velocity and mass columns) are
// exact no-ops of that chain and are skipped.
template <int N>
__device__ __forceinline__ void dqdt_op(Sys<N>& s, Work<N>& w, double div) {
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) {
      int vr = 3 * b + k;
      double acc = 0.0;
      for (int d = 0; d < N; d++)
        for (int p = 0; p < 3; p++) acc = fma(OPX(vr, 4 * d + p), s.dqdt[7 * d + p], acc);
      double dq = (div != 1.0) ? w.dqop[vr] / div : w.dqop[vr];
      s.dqdt[7 * b + 3 + k] = s.dqdt[7 * b + 3 + k] + (dq + acc);
    }
}

__device__ __forceinline__ void put_op(const Rec& rec, int off, const double* op, int n) {
  for (int q = 0; q < n; q++) rec.put(off + q, op[q]);
}

// phic! (ahl21.jl:392-552 / ahl21_no_grad.jl:62-104): corrector for kick pairs
template <int N>
__device__ void phic(Sys<N>& s, Work<N>& w, double h, uint64_t kick) {
  for (int q = 0; q < 3 * N; q++) w.a[q] = 0.0;
  for (int q = 0; q < 12 * N * N; q++) { w.dadq[q] = 0.0; w.op[q] = 0.0; }
  for (int q = 0; q < 3 * N; q++) w.dqop[q] = 0.0;
  if (!kick) return;
  double coeff = h * h * h / 36.0 * GNEWT;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (!((kick >> pair_bit(i, j, N)) & 1)) continue;
      double rij[3];
      for (int k = 0; k < 3; k++) rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      double r2inv = 1.0 / (rij[0] * rij[0] + rij[1] * rij[1] + rij[2] * rij[2]);
      double r3inv = r2inv * sqrt(r2inv);
      for (int k = 0; k < 3; k++) {
        double fac = GNEWT * rij[k] * r3inv;
        double facv = fac * 2.0 * h / 3.0;
        kahan(s.v[3 * i + k], s.ve[3 * i + k], (-s.m[j]) * facv);
        kahan(s.v[3 * j + k], s.ve[3 * j + k], s.m[i] * facv);
        w.a[3 * i + k] = w.a[3 * i + k] - s.m[j] * fac;
        w.a[3 * j + k] = w.a[3 * j + k] + s.m[i] * fac;
        w.dqop[3 * i + k] = w.dqop[3 * i + k] - 1.0 / h * s.m[j] * facv;
        w.dqop[3 * j + k] = w.dqop[3 * j + k] + 1.0 / h * s.m[i] * facv;
        OPX(3 * i + k, 4 * j + 3) -= facv;
        OPX(3 * j + k, 4 * i + 3) += facv;
        facv = facv * (3.0 * r2inv);
        for (int p = 0; p < 3; p++) {
          OPX(3 * i + k, 4 * i + p) += facv * s.m[j] * rij[p];
          OPX(3 * i + k, 4 * j + p) -= facv * s.m[j] * rij[p];
          OPX(3 * j + k, 4 * j + p) += facv * s.m[i] * rij[p];
          OPX(3 * j + k, 4 * i + p) -= facv * s.m[i] * rij[p];
        }
        facv = 2.0 * h / 3.0 * GNEWT * r3inv;
        OPX(3 * i + k, 4 * i + k) -= facv * s.m[j];
        OPX(3 * i + k, 4 * j + k) += facv * s.m[j];
        OPX(3 * j + k, 4 * j + k) -= facv * s.m[i];
        OPX(3 * j + k, 4 * i + k) += facv * s.m[i];
        DAX(3 * i + k, 4 * j + 3) -= fac;
        DAX(3 * j + k, 4 * i + 3) += fac;
        fac = fac * (3.0 * r2inv);
        for (int p = 0; p < 3; p++) {
          DAX(3 * i + k, 4 * i + p) += fac * s.m[j] * rij[p];
          DAX(3 * i + k, 4 * j + p) -= fac * s.m[j] * rij[p];
          DAX(3 * j + k, 4 * j + p) += fac * s.m[i] * rij[p];
          DAX(3 * j + k, 4 * i + p) -= fac * s.m[i] * rij[p];
        }
        fac = GNEWT * r3inv;
        DAX(3 * i + k, 4 * i + k) -= fac * s.m[j];
        DAX(3 * i + k, 4 * j + k) += fac * s.m[j];
        DAX(3 * j + k, 4 * j + k) -= fac * s.m[i];
        DAX(3 * j + k, 4 * i + k) += fac * s.m[i];
      }
    }
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (!((kick >> pair_bit(i, j, N)) & 1)) continue;
      double rij[3], aij[3];
      for (int k = 0; k < 3; k++) {
        aij[k] = w.a[3 * i + k] - w.a[3 * j + k];
        rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      }
      for (int q = 0; q < 4 * N; q++) w.dot[q] = 0.0;
      for (int di = 0; di < N; di++)
        for (int p = 0; p < 4; p++)
          for (int k = 0; k < 3; k++)
            w.dot[4 * di + p] += rij[k] * (DAX(3 * i + k, 4 * di + p) - DAX(3 * j + k, 4 * di + p));
      double r2 = rij[0] * rij[0] + rij[1] * rij[1] + rij[2] * rij[2];
      double r1 = sqrt(r2);
      double ardot = aij[0] * rij[0] + aij[1] * rij[1] + aij[2] * rij[2];
      double fac1 = coeff / (r2 * r2 * r1);
      double fac2 = 3.0 * ardot;
      for (int k = 0; k < 3; k++) {
        double fac = fac1 * (rij[k] * fac2 - r2 * aij[k]);
        kahan(s.v[3 * i + k], s.ve[3 * i + k], s.m[j] * fac);
        kahan(s.v[3 * j + k], s.ve[3 * j + k], (-s.m[i]) * fac);
        w.dqop[3 * i + k] = w.dqop[3 * i + k] + 3.0 / h * s.m[j] * fac;
        w.dqop[3 * j + k] = w.dqop[3 * j + k] - 3.0 / h * s.m[i] * fac;
        OPX(3 * i + k, 4 * j + 3) += fac;
        OPX(3 * j + k, 4 * i + 3) -= fac;
        fac = fac * (5.0 / r2);
        for (int p = 0; p < 3; p++) {
          OPX(3 * i + k, 4 * i + p) -= fac * s.m[j] * rij[p];
          OPX(3 * i + k, 4 * j + p) += fac * s.m[j] * rij[p];
          OPX(3 * j + k, 4 * j + p) -= fac * s.m[i] * rij[p];
          OPX(3 * j + k, 4 * i + p) += fac * s.m[i] * rij[p];
        }
        fac = fac1 * fac2;
        OPX(3 * i + k, 4 * i + k) += fac * s.m[j];
        OPX(3 * i + k, 4 * j + k) -= fac * s.m[j];
        OPX(3 * j + k, 4 * j + k) += fac * s.m[i];
        OPX(3 * j + k, 4 * i + k) -= fac * s.m[i];
        fac = -2.0 * fac1 * aij[k];
        for (int p = 0; p < 3; p++) {
          double fac3 = fac * rij[p] + fac1 * 3.0 * rij[k] * aij[p];
          OPX(3 * i + k, 4 * i + p) += s.m[j] * fac3;
          OPX(3 * i + k, 4 * j + p) -= s.m[j] * fac3;
          OPX(3 * j + k, 4 * j + p) += s.m[i] * fac3;
          OPX(3 * j + k, 4 * i + p) -= s.m[i] * fac3;
        }
        fac = (-fac1) * r2;
        for (int di = 0; di < N; di++) {
          for (int p = 0; p < 3; p++) {
            OPX(3 * i + k, 4 * di + p) += fac * s.m[j] * (DAX(3 * i + k, 4 * di + p) - DAX(3 * j + k, 4 * di + p));
            OPX(3 * j + k, 4 * di + p) -= fac * s.m[i] * (DAX(3 * i + k, 4 * di + p) - DAX(3 * j + k, 4 * di + p));
          }
          OPX(3 * i + k, 4 * di + 3) += fac * s.m[j] * (DAX(3 * i + k, 4 * di + 3) - DAX(3 * j + k, 4 * di + 3));
          OPX(3 * j + k, 4 * di + 3) -= fac * s.m[i] * (DAX(3 * i + k, 4 * di + 3) - DAX(3 * j + k, 4 * di + 3));
        }
        fac = 3.0 * fac1 * rij[k];
        for (int di = 0; di < N; di++) {
          for (int p = 0; p < 3; p++) {
            OPX(3 * i + k, 4 * di + p) += fac * s.m[j] * w.dot[4 * di + p];
            OPX(3 * j + k, 4 * di + p) -= fac * s.m[i] * w.dot[4 * di + p];
          }
          OPX(3 * i + k, 4 * di + 3) += fac * s.m[j] * w.dot[4 * di + 3];
          OPX(3 * j + k, 4 * di + 3) -= fac * s.m[i] * w.dot[4 * di + 3];
        }
      }
    }
}

// A pair's terms of the steps without gradient, each rounded as the reference's
// expressions are: G r / r^3 of the correctors (ahl21_no_grad.jl:120-127)
__device__ __forceinline__ double norm2(const double* r) { return r[0] * r[0] + r[1] * r[1] + r[2] * r[2]; }
__device__ __forceinline__ void phis_accel(const double* rij, double r2, double r1, double* f) {
  const double fac2 = GNEWT / (r2 * r1);
#pragma unroll
  for (int k = 0; k < 3; k++) f[k] = fac2 * rij[k];
}
// the corrections (ahl21_no_grad.jl:140-152; with mij = 0 those of :88-99)
__device__ __forceinline__ void phis_corr(const double* rij, double r2, double r1, const double* aij, double mij,
                                          double coeff, double* f) {
  const double ardot = aij[0] * rij[0] + aij[1] * rij[1] + aij[2] * rij[2];
  const double fac1 = coeff / (r2 * r2 * r1);
  const double fac2 = mij != 0.0 ? 2.0 * GNEWT * mij / r1 + 3.0 * ardot : 3.0 * ardot;
#pragma unroll
  for (int k = 0; k < 3; k++) f[k] = fac1 * (rij[k] * fac2 - r2 * aij[k]);
}
// 1 / r^3 of a kick pair (ahl21_no_grad.jl:42-43)
__device__ __forceinline__ double kick_r3inv(const double* rij) {
  const double r2inv = 1.0 / norm2(rij);
  return r2inv * sqrt(r2inv);
}
__device__ __forceinline__ double phis_coeff(double h) {  // alpha = 2 (ahl21.jl:47)
  return 2.0 * (h * h * h) / 96.0 * 2.0 * GNEWT;
}
__device__ __forceinline__ double phic_coeff(double h) { return h * h * h / 36.0 * GNEWT; }

// phisalpha! (ahl21.jl:558-700 / ahl21_no_grad.jl:110-158) for Kepler pairs,
// one pair at a time: the accelerations, then the velocity corrections.
template <int N>
__device__ __forceinline__ void phis_accel_pair(const Sys<N>& s, double* a, int i, int j) {
  double rij[3], f[3];
#pragma unroll
  for (int k = 0; k < 3; k++) rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
  const double r2 = norm2(rij);
  phis_accel(rij, r2, sqrt(r2), f);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    a[3 * i + k] = a[3 * i + k] - s.m[j] * f[k];
    a[3 * j + k] = a[3 * j + k] + s.m[i] * f[k];
  }
}
template <int N>
__device__ __forceinline__ void phis_kick_pair(Sys<N>& s, const double* a, int i, int j, double mij, double coeff) {
  double rij[3], aij[3], f[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    aij[k] = a[3 * i + k] - a[3 * j + k];
    rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
  }
  const double r2 = norm2(rij);
  phis_corr(rij, r2, sqrt(r2), aij, mij, coeff, f);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    kahan(s.v[3 * i + k], s.ve[3 * i + k], s.m[j] * f[k]);
    kahan(s.v[3 * j + k], s.ve[3 * j + k], (-s.m[i]) * f[k]);
  }
}
template <int N>
__device__ __forceinline__ void phisalpha(Sys<N>& s, double* a, double h, uint64_t kick) {
  const double coeff = phis_coeff(h);
#pragma unroll
  for (int q = 0; q < 3 * N; q++) a[q] = 0.0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if (!((kick >> pair_bit(i, j, N)) & 1)) phis_accel_pair<N>(s, a, i, j);
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if (!((kick >> pair_bit(i, j, N)) & 1)) phis_kick_pair<N>(s, a, i, j, s.m[i] + s.m[j], coeff);
}

// kickfast! without gradient (ahl21_no_grad.jl:35-56): kicks over h between the
// pairs of the mask.
template <int N>
__device__ __forceinline__ void plain_kick(Sys<N>& s, double h, uint64_t kick) {
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (!((kick >> pair_bit(i, j, N)) & 1)) continue;
      double rij[3];
#pragma unroll
      for (int k = 0; k < 3; k++) rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      const double fac2 = h * GNEWT * kick_r3inv(rij);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const double fac = fac2 * rij[k];
        kahan(s.v[3 * i + k], s.ve[3 * i + k], (-s.m[j]) * fac);
        kahan(s.v[3 * j + k], s.ve[3 * j + k], s.m[i] * fac);
      }
    }
}
// phic! without gradient (ahl21_no_grad.jl:62-104): a kick over 2h/3 and the
// correction, between the pairs of the mask.
template <int N>
__device__ __forceinline__ void plain_phic(Sys<N>& s, double* a, double h, uint64_t kick) {
#pragma unroll
  for (int q = 0; q < 3 * N; q++) a[q] = 0.0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (!((kick >> pair_bit(i, j, N)) & 1)) continue;
      double rij[3];
#pragma unroll
      for (int k = 0; k < 3; k++) rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      const double r3inv = kick_r3inv(rij);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const double fac = GNEWT * rij[k] * r3inv, facv = fac * 2.0 * h / 3.0;
        kahan(s.v[3 * i + k], s.ve[3 * i + k], (-s.m[j]) * facv);
        kahan(s.v[3 * j + k], s.ve[3 * j + k], s.m[i] * facv);
        a[3 * i + k] = a[3 * i + k] - s.m[j] * fac;
        a[3 * j + k] = a[3 * j + k] + s.m[i] * fac;
      }
    }
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if ((kick >> pair_bit(i, j, N)) & 1) phis_kick_pair<N>(s, a, i, j, 0.0, phic_coeff(h));
}

// The corrector's operator (jac_phi, ahl21.jl:558-700) for Kepler pairs: its
// four columns of body d (position and mass), rows 3b + k, added to
// acc[4 (3b + k) + p].  x: the positions at the corrector, a: the
// accelerations phisalpha formed there.
//
// The velocity correction of pair (i, j) is m_j F, -m_i F with
// F = fac1 (r fac2 - r^2 (a_i - a_j)), so a column is E (r's own change) plus
// M (a_i - a_j)' with M = fac1 (3 r r^T - r^2), and only a_d and the pairs with
// d enter the accelerations' change: one lane per (step, body) needs no
// 3N x 4N array and no other lane, about 110 FP64 instructions a pair.
// POS = false: the mass column alone.
template <int N, bool POS = true>
__device__ __forceinline__ void phi_columns(const double* x, const double* a, const double* m, double h,
                                            uint64_t kick, int d, double* acc) {
  // change of each body's acceleration by x_d (symmetric: xx, xy, xz, yy, yz, zz) and by m_d
  double blk[N][9];
  double own[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double md = m[d];
  constexpr int P0 = POS ? 0 : 3;
#pragma unroll 1
  for (int i = 0; i < N; i++) {
#pragma unroll
    for (int q = 0; q < 9; q++) blk[i][q] = 0.0;
    if (i == d || ((kick >> (i < d ? pair_bit(i, d, N) : pair_bit(d, i, N))) & 1)) continue;
    double r[3];
#pragma unroll
    for (int k = 0; k < 3; k++) r[k] = x[3 * i + k] - x[3 * d + k];
    const double ri = rsqrt_fast(fma(r[2], r[2], fma(r[1], r[1], r[0] * r[0])));
    const double ri2 = ri * ri, f2 = (GNEWT * ri) * ri2, g5 = 3.0 * f2 * ri2;
    const double gx = g5 * r[0], gy = g5 * r[1], gz = g5 * r[2];
    const double T[6] = {fma(gx, r[0], -f2), gx * r[1], gx * r[2], fma(gy, r[1], -f2), gy * r[2], fma(gz, r[2], -f2)};
#pragma unroll
    for (int q = 0; q < (POS ? 6 : 0); q++) {
      blk[i][q] = -(md * T[q]);
      own[q] = fma(m[i], T[q], own[q]);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) blk[i][6 + k] = -(f2 * r[k]);
  }
#pragma unroll
  for (int q = 0; q < 6; q++) blk[d][q] = own[q];
  const double coeff = phis_coeff(h);
#pragma unroll 1
  for (int i = 0; i < N - 1; i++)
#pragma unroll 1
    for (int j = i + 1; j < N; j++) {
      if ((kick >> pair_bit(i, j, N)) & 1) continue;
      double r[3], aij[3], D[9];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        r[k] = x[3 * i + k] - x[3 * j + k];
        aij[k] = a[3 * i + k] - a[3 * j + k];
      }
#pragma unroll
      for (int q = P0 ? 6 : 0; q < 9; q++) D[q] = blk[i][q] - blk[j][q];
      const double r2 = fma(r[2], r[2], fma(r[1], r[1], r[0] * r[0]));
      const double ri = rsqrt_fast(r2), ri2 = ri * ri;
      const double fac1 = (coeff * ri) * (ri2 * ri2), f3 = 3.0 * fac1, fr = fac1 * r2;
      double G[3][4];
      const double col[4][3] = {{D[0], D[1], D[2]}, {D[1], D[3], D[4]}, {D[2], D[4], D[5]}, {D[6], D[7], D[8]}};
#pragma unroll
      for (int p = P0; p < 4; p++) {
        const double c = f3 * fma(r[2], col[p][2], fma(r[1], col[p][1], r[0] * col[p][0]));
#pragma unroll
        for (int k = 0; k < 3; k++) G[k][p] = fma(r[k], c, -(fr * col[p][k]));
      }
      if (d == i || d == j) {
        const double mij = m[i] + m[j];
        const double ardot = fma(aij[2], r[2], fma(aij[1], r[1], aij[0] * r[0]));
        const double gri = (2.0 * GNEWT) * ri, fac2 = fma(gri, mij, 3.0 * ardot);
        const double sg = (d == i) ? 1.0 : -1.0;
        const double q5 = -5.0 * ri2, q3 = gri * ri2 * mij, diag = sg * (fac1 * fac2), fg = fac1 * gri;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const double F = fac1 * fma(r[k], fac2, -(r2 * aij[k]));
          const double e = sg * fma(q5, F, -(fac1 * fma(q3, r[k], 2.0 * aij[k]))), f = sg * (f3 * r[k]);
#pragma unroll
          for (int p = P0; p < 3; p++) G[k][p] = fma(f, aij[p], fma(e, r[p], G[k][p]));
          if (POS) G[k][k] = G[k][k] + diag;
          G[k][3] = fma(fg, r[k], G[k][3]);
          acc[12 * (d == i ? j : i) + 4 * k + 3] += (d == i) ? -F : F;
        }
      }
      const double mi = -m[i], mj = m[j];
#pragma unroll
      for (int k = 0; k < 3; k++)
#pragma unroll
        for (int p = P0; p < 4; p++) {
          acc[12 * i + 4 * k + p] = fma(mj, G[k][p], acc[12 * i + 4 * k + p]);
          acc[12 * j + 4 * k + p] = fma(mi, G[k][p], acc[12 * j + 4 * k + p]);
        }
    }
}

// The same for every body, onto w.op, and d(v)/dh of the corrector, onto w.dqop.
template <int N>
__device__ void phisalpha_operator(const Sys<N>& s, Work<N>& w, double h, uint64_t kick) {
  for (int d = 0; d < N; d++) {
    double acc[12 * N];
    for (int q = 0; q < 12 * N; q++) acc[q] = 0.0;
    phi_columns<N>(s.x, w.a, s.m, h, kick, d, acc);
    for (int r = 0; r < 3 * N; r++)
      for (int p = 0; p < 4; p++) OPX(r, 4 * d + p) += acc[4 * r + p];
  }
  const double coeff = phis_coeff(h), hi3 = 3.0 / h;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if ((kick >> pair_bit(i, j, N)) & 1) continue;
      double rij[3], aij[3], f[3];
      for (int k = 0; k < 3; k++) {
        aij[k] = w.a[3 * i + k] - w.a[3 * j + k];
        rij[k] = s.x[3 * i + k] - s.x[3 * j + k];
      }
      const double r2 = norm2(rij);
      phis_corr(rij, r2, sqrt(r2), aij, s.m[i] + s.m[j], coeff, f);
      for (int k = 0; k < 3; k++) {
        w.dqop[3 * i + k] = fma(hi3 * s.m[j], f[k], w.dqop[3 * i + k]);
        w.dqop[3 * j + k] = fma(-hi3 * s.m[i], f[k], w.dqop[3 * j + k]);
      }
    }
}

// Writes one solved pair's capture (pair_record_from_capture reads it).
__device__ __forceinline__ void put_capture(const Rec& cap, int coff, const double* x0, const double* v0,
                                            const KepParams& P) {
  const double pv[PCAP] = {x0[0], x0[1], x0[2], v0[0],  v0[1], v0[2], P.gamma, P.g2, P.g3,
                           P.r0,  P.r0inv, P.rinv, P.beta, P.eta, P.fm1, P.gmh, P.dfdt, P.dgdtm1};
#pragma unroll
  for (int q = 0; q < PCAP; q++) cap.put(coff + q, pv[q]);
}

// kepler_driftij_gamma! without Jacobian (ahl21_no_grad.jl:192-212).  P and
// delxv are left for the caller's Jacobian; false for a pair without mass.
template <int N, bool DRIFT_FIRST>
__device__ __forceinline__ bool kepler_pair(Sys<N>& s, int i, int j, double h2, const Rec& cap, int coff, double* x0,
                                            double* v0, KepParams& P, double* delxv) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    x0[k] = s.x[3 * i + k] - s.x[3 * j + k];
    v0[k] = s.v[3 * i + k] - s.v[3 * j + k];
  }
  const double mij = s.m[i] + s.m[j];
  const double gm = GNEWT * mij;
  if (gm == 0.0) {
    if (cap.p) cap.put(coff + PCAP_RINV, 0.0);  // a pair that keeps the stale jac_ij
    return false;
  }
  kep_solve<DRIFT_FIRST>(x0, v0, gm, h2, delxv, P);
  if (cap.p) put_capture(cap, coff, x0, v0, P);
  const double mijinv = 1.0 / mij;
  const double mi = s.m[i] * mijinv, mj = s.m[j] * mijinv;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    kahan(s.x[3 * i + k], s.xe[3 * i + k], mj * delxv[k]);
    kahan(s.x[3 * j + k], s.xe[3 * j + k], (-mi) * delxv[k]);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    kahan(s.v[3 * i + k], s.ve[3 * i + k], mj * delxv[3 + k]);
    kahan(s.v[3 * j + k], s.ve[3 * j + k], (-mi) * delxv[3 + k]);
  }
  return true;
}
template <int N, bool DRIFT_FIRST>
__device__ __forceinline__ void kepler_pair(Sys<N>& s, int i, int j, double h2, const Rec& cap, int coff) {
  double x0[3], v0[3], delxv[6];
  KepParams P;
  kepler_pair<N, DRIFT_FIRST>(s, i, j, h2, cap, coff, x0, v0, P, delxv);
}

// The same with the block update of ahl21.jl:31-42 on dq/dt (ahl21.jl:706-760).
template <int N, bool DRIFT_FIRST>
__device__ void kepler_pair_grad(Sys<N>& s, Work<N>& w, int i, int j, double h2, const Rec& rec, int roff) {
  double x0[3], v0[3], delxv[6];
  KepParams P;
  if (kepler_pair<N, DRIFT_FIRST>(s, i, j, h2, Rec{nullptr, 0}, 0, x0, v0, P, delxv)) {
    const double mijinv = rcp_fast(s.m[i] + s.m[j]);
    const double mi = s.m[i] * mijinv, mj = s.m[j] * mijinv;
    {
      KepDeriv D;
      double dh[6];
      kep_derivatives<DRIFT_FIRST, true>(P, D);
      kep_block<DRIFT_FIRST>(P, D, x0, v0, w.lk, w.lpsi);
      kep_by_h<DRIFT_FIRST>(P, D, x0, v0, dh);
      w.lmi = mi;
      w.lmj = mj;
      for (int r = 0; r < 6; r++) {
        w.lb[r] = mijinv * delxv[r];
        w.ldq[r] = mj * dh[r];
        w.ldq[7 + r] = (-mi) * dh[r];
      }
      w.ldq[6] = w.ldq[13] = 0.0;
    }
  }
  if (rec.p) {
    for (int q = 0; q < 36; q++) rec.put(roff + q, w.lk[q]);
    rec.put(roff + PREC_MI, w.lmi);
    rec.put(roff + PREC_MJ, w.lmj);
    for (int q = 0; q < 6; q++) {
      rec.put(roff + PREC_PSI + q, w.lpsi[q]);
      rec.put(roff + PREC_B + q, w.lb[q]);
    }
  }
  {
    // d.dqdt_ij .*= 1/2; d.dqdt_ij .+= dqdt_tmp1 .+ jac_ij * dqdt_tmp1 (ahl21.jl:38-40)
    double t1[14];
    for (int q = 0; q < 7; q++) {
      t1[q] = s.dqdt[7 * i + q];
      t1[7 + q] = s.dqdt[7 * j + q];
    }
    for (int q = 0; q < 14; q++) w.ldq[q] = w.ldq[q] * 0.5;
    for (int r = 0; r < 6; r++) {
      double ai = 0.0, aj = 0.0;
      for (int l = 0; l < 6; l++) {
        double kij = w.lmj * w.lk[r * 6 + l];
        double kji = w.lmi * w.lk[r * 6 + l];
        ai = fma(kij, t1[l], ai);
        aj = fma(-kji, t1[l], aj);
      }
      for (int l = 0; l < 6; l++) {
        double kij = w.lmj * w.lk[r * 6 + l];
        double kji = w.lmi * w.lk[r * 6 + l];
        ai = fma(-kij, t1[7 + l], ai);
        aj = fma(kji, t1[7 + l], aj);
      }
      w.ldq[r] = w.ldq[r] + (t1[r] + ai);
      w.ldq[7 + r] = w.ldq[7 + r] + (t1[7 + r] + aj);
    }
    w.ldq[6] = w.ldq[6] + (t1[6] + 0.0);
    w.ldq[13] = w.ldq[13] + (t1[13] + 0.0);
    for (int q = 0; q < 7; q++) {
      s.dqdt[7 * i + q] = w.ldq[q];
      s.dqdt[7 * j + q] = w.ldq[7 + q];
    }
  }
}

// One AHL21 step with its gradient (ahl21.jl:5-95): x, v, dq/dt as the reference
// forms it, and the operator record at rec.
template <int N>
__device__ __noinline__ void ahl21_step(Sys<N>& s, Work<N>& w, double h, uint64_t kick, const Rec& rec) {
  const double h2 = 0.5 * h, h6 = h / 6.0;
  reset_last(w);
  for (int q = 0; q < 7 * N; q++) s.dqdt[q] = 0.0;
  int roff = 0;
  if (kick) {
    kickfast<N>(s, w, h6, kick);
    dqdt_op(s, w, 6.0);
    put_op(rec, roff, w.op, op_size(N));
    roff += op_size(N);
  }
  drift(s, h2);
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) s.dqdt[7 * b + k] = 0.5 * s.v[3 * b + k] + h2 * s.dqdt[7 * b + 3 + k];
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if ((kick >> pair_bit(i, j, N)) & 1) continue;
      kepler_pair_grad<N, true>(s, w, i, j, h2, rec, roff);
      roff += PREC;
    }
  phic<N>(s, w, h, kick);
  phisalpha<N>(s, w.a, h, kick);  // moves v alone: the operator below is that of the same positions
  phisalpha_operator<N>(s, w, h, kick);
  dqdt_op(s, w, 1.0);
  put_op(rec, roff, w.op, op_size(N));
  roff += op_size(N);
  for (int i = N - 2; i >= 0; i--)
    for (int j = N - 1; j > i; j--) {
      if ((kick >> pair_bit(i, j, N)) & 1) continue;
      kepler_pair_grad<N, false>(s, w, i, j, h2, rec, roff);
      roff += PREC;
    }
  drift(s, h2);
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++)
      s.dqdt[7 * b + k] = s.dqdt[7 * b + k] + (0.5 * s.v[3 * b + k] + h2 * s.dqdt[7 * b + 3 + k]);
  if (kick) {
    kickfast<N>(s, w, h6, kick);
    dqdt_op(s, w, 6.0);
    put_op(rec, roff, w.op, op_size(N));
  }
}

// The same step without gradient (ahl21_no_grad.jl:6-18): x and v alone, a the
// accelerations at the corrector.  cap, xs, vs: where the captures and
// snapshots go (snap_count) and, for dq/dt, v at the first drift and at the
// second (3N each); p == nullptr: nowhere.
template <int N>
__device__ __forceinline__ void plain_step(Sys<N>& s, double* a, double h, uint64_t kick, const Rec& cap,
                                           const Rec& xs, const Rec& vs) {
  const double h2 = 0.5 * h;
  int slot = 0;
  if (kick) {
    if (xs.p)
      for (int q = 0; q < 3 * N; q++) xs.put(3 * N + q, s.x[q]);
    plain_kick<N>(s, h / 6.0, kick);
  }
  if (vs.p)
    for (int q = 0; q < 3 * N; q++) vs.put(q, s.v[q]);
  drift(s, h2);
#pragma unroll 1
  for (int i = 0; i < N - 1; i++)
#pragma unroll 1
    for (int j = i + 1; j < N; j++)
      if (!((kick >> pair_bit(i, j, N)) & 1)) kepler_pair<N, true>(s, i, j, h2, cap, PCAP * slot++);
  if (xs.p)
    for (int q = 0; q < 3 * N; q++) xs.put(q, s.x[q]);
  if (kick) plain_phic<N>(s, a, h, kick);
  phisalpha<N>(s, a, h, kick);
  if (xs.p && !kick)
    for (int q = 0; q < 3 * N; q++) xs.put(3 * N + q, a[q]);
#pragma unroll 1
  for (int i = N - 2; i >= 0; i--)
#pragma unroll 1
    for (int j = N - 1; j > i; j--)
      if (!((kick >> pair_bit(i, j, N)) & 1)) kepler_pair<N, false>(s, i, j, h2, cap, PCAP * slot++);
  if (vs.p)
    for (int q = 0; q < 3 * N; q++) vs.put(3 * N + q, s.v[q]);
  drift(s, h2);
  if (kick) {
    if (xs.p)
      for (int q = 0; q < 3 * N; q++) xs.put(6 * N + q, s.x[q]);
    plain_kick<N>(s, h / 6.0, kick);
  }
}

// g! and gd! (src/transits/timing.jl:141-150) for transited body i and
// occultor j.
template <int N>
__device__ __forceinline__ double gsky(const Sys<N>& s, int i, int j) {
  return (s.x[3 * j] - s.x[3 * i]) * (s.v[3 * j] - s.v[3 * i]) +
         (s.x[3 * j + 1] - s.x[3 * i + 1]) * (s.v[3 * j + 1] - s.v[3 * i + 1]);
}
template <int N>
__device__ __forceinline__ double gdot(const Sys<N>& s, int i, int j) {
  const double* q = s.dqdt;
  return ((s.x[3 * j] - s.x[3 * i]) * (q[7 * j + 3] - q[7 * i + 3]) +
          (s.x[3 * j + 1] - s.x[3 * i + 1]) * (q[7 * j + 4] - q[7 * i + 4]) +
          (s.v[3 * j] - s.v[3 * i]) * (q[7 * j + 0] - q[7 * i + 0]) +
          (s.v[3 * j + 1] - s.v[3 * i + 1]) * (q[7 * j + 1] - q[7 * i + 1]));
}

// detect_transits! (timing.jl:3-28) for occultor slot o after step kk of the
// chunk: g's sign change with the occultor in front queues a search from a copy
// of this state (transit_kernel runs it, so that no other system of the warp
// waits).  gsave, count: the system's N entries.
template <int N>
__device__ __forceinline__ void detect_transit(const GroupArgs& g, const Sys<N>& st, int s, int kk, int o, int ti,
                                               int ntt, double hI, double t, double* gsave, long long* count) {
  const int ib = (o < ti) ? o : o + 1, S = g.S;
  const double gi = gsky(st, ib, ti), before = gsave[ib];
  gsave[ib] = gi;
  if (g.grad) g.tflag[(size_t)(kk * (N - 1) + o) * S + s] = -1;
  if (!(gi > 0.0 && before < 0.0)) return;
  const double xi = st.x[3 * ib], yi = st.x[3 * ib + 1], zi = st.x[3 * ib + 2];
  const double ri = sqrt(xi * xi + yi * yi + zi * zi);
  if (!(-zi > 0.25 * ri && ri < 1e12)) return;
  count[ib] += 1;
  if (count[ib] > ntt) {
    atomicOr(g.status + s, NBG_STATUS_NTT_OVERFLOW);
    return;
  }
  const int idx = atomicAdd(g.task_count, 1);
  if (idx >= g.task_cap) return;  // the capacity is the number of (step, occultor, system) slots
  double* tf = g.task_f + (size_t)idx * (12 * N + 2);
  for (int q = 0; q < 3 * N; q++) {
    tf[q] = st.x[q];
    tf[3 * N + q] = st.v[q];
    tf[6 * N + q] = st.xe[q];
    tf[9 * N + q] = st.ve[q];
  }
  tf[12 * N] = -gi * hI / (gi - before);  // first estimate (timing.jl:20)
  tf[12 * N + 1] = t;
  int* tk = g.task_i + 3 * idx;
  tk[0] = s;
  tk[1] = kk * (N - 1) + o;
  tk[2] = (int)(count[ib] - 1);
}

// u <- u + A^T u for the compact operator block A (velocity rows x position
// and mass columns); reads the record at roff.
template <int N>
__device__ void adj_op(double* u, const Rec& rec, int roff) {
  double add[4 * N];
  for (int d = 0; d < N; d++)
    for (int p = 0; p < 4; p++) {
      double acc = 0.0;
      for (int b = 0; b < N; b++)
        for (int k = 0; k < 3; k++) acc = fma(rec.get(roff + (3 * b + k) * (4 * N) + 4 * d + p), u[7 * b + 3 + k], acc);
      add[4 * d + p] = acc;
    }
  for (int d = 0; d < N; d++) {
    for (int p = 0; p < 3; p++) u[7 * d + p] = u[7 * d + p] + add[4 * d + p];
    u[7 * d + 6] = u[7 * d + 6] + add[4 * d + 3];
  }
}

// u <- u + A^T u for one Kepler pair record (the transpose of the factored
// jac_ij update the consumer applies).
__device__ __forceinline__ void adj_pair(double* u, int i, int j, const Rec& rec, int roff) {
  const double mi = rec.get(roff + PREC_MI), mj = rec.get(roff + PREC_MJ);
  double z[6], psi = 0.0, bi = 0.0, bj = 0.0;
#pragma unroll
  for (int r = 0; r < 6; r++) {
    const double ui = u[7 * i + r], uj = u[7 * j + r], b = rec.get(roff + PREC_B + r);
    z[r] = fma(mj, ui, -(mi * uj));
    psi = fma(rec.get(roff + PREC_PSI + r), z[r], psi);
    bi = fma(b, uj, bi);
    bj = fma(b, ui, bj);
  }
#pragma unroll
  for (int l = 0; l < 6; l++) {
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < 6; r++) acc = fma(rec.get(roff + r * 6 + l), z[r], acc);
    u[7 * i + l] = u[7 * i + l] + acc;
    u[7 * j + l] = u[7 * j + l] - acc;
  }
  u[7 * i + 6] = u[7 * i + 6] + (psi - bi);
  u[7 * j + 6] = u[7 * j + 6] + (psi + bj);
}

// Adjoint of one recorded step: u^T <- u^T S where S is the step's map on
// jac_step (ahl21.jl:5-95): (I+K2)(I+D)prod_bwd(I+A)(I+Phi)prod_fwd(I+A)(I+D+K1).
// The first kick's product is formed before the first drift and added after
// it (ahl21.jl:16-23), hence the I + D + K1 factor.
template <int N>
__device__ void adjoint_step(double* u, double h, uint64_t kick, const Rec& rec) {
  const double h2 = 0.5 * h;
  int npk = 0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if (!((kick >> pair_bit(i, j, N)) & 1)) npk++;
  int off_k1 = 0;
  int off_fwd = kick ? op_size(N) : 0;
  int off_phi = off_fwd + npk * PREC;
  int off_bwd = off_phi + op_size(N);
  int off_k2 = off_bwd + npk * PREC;
  if (kick) adj_op<N>(u, rec, off_k2);
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) u[7 * b + 3 + k] = u[7 * b + 3 + k] + h2 * u[7 * b + k];
  // backward sweep was applied in order (N-2..0, N-1..i+1); undo in reverse
  {
    int q = npk - 1;
    for (int i = 0; i < N - 1; i++)
      for (int j = i + 1; j < N; j++) {
        if ((kick >> pair_bit(i, j, N)) & 1) continue;
        adj_pair(u, i, j, rec, off_bwd + q * PREC);
        q--;
      }
  }
  adj_op<N>(u, rec, off_phi);
  {
    int q = npk - 1;
    for (int i = N - 2; i >= 0; i--)
      for (int j = N - 1; j > i; j--) {
        if ((kick >> pair_bit(i, j, N)) & 1) continue;
        adj_pair(u, i, j, rec, off_fwd + q * PREC);
        q--;
      }
  }
  if (kick) {
    // both terms of I + D + K1 act on the same u: D^T reads the position
    // entries, K1^T reads the velocity entries and writes positions/masses.
    double ux[3 * N];
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) ux[3 * b + k] = u[7 * b + k];
    adj_op<N>(u, rec, off_k1);
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) u[7 * b + 3 + k] = u[7 * b + 3 + k] + h2 * ux[3 * b + k];
  } else {
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) u[7 * b + 3 + k] = u[7 * b + 3 + k] + h2 * u[7 * b + k];
  }
}

#undef OPX
#undef DAX

}  // namespace nbg
