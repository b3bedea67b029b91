// nbg_operators.cuh -- builds the step operator records from the parameters
// the orbit producer captured, in parallel over (step, pair, system).
//
// The producer advances x, v only (the arithmetic of ahl21_no_grad.jl, bitwise
// the x, v of the gradient step) and captures, per Kepler pair, x0, v0 and the
// values of its solve (put_capture), plus the positions and accelerations at
// the correctors and kicks.  Everything else kepler_driftij_gamma!,
// phic!/phisalpha! and kickfast! compute for the Jacobian depends only on
// those values, so it runs here, off the producer's sequential chain:
//   * compute_jacobian_gamma! (ahl21.jl:896-1139) and the jac_ij assembly
//     (ahl21.jl:727-750) per pair;
//   * jac_phi (ahl21.jl:392-700) and jac_kick (ahl21.jl:337-386) per step.
#pragma once
#include "nbg_orbit.cuh"

namespace nbg {

// Bodies (i, j) of Kepler-pair slot q of a step: slots 0..npk-1 follow the
// forward sweep (i ascending, j ascending), npk..2npk-1 the backward sweep.
template <int N>
__device__ __forceinline__ void pair_of_slot(int q, int npk, uint64_t kick, int* pi, int* pj) {
  int c = 0;
  if (q < npk) {
    for (int i = 0; i < N - 1; i++)
      for (int j = i + 1; j < N; j++) {
        if ((kick >> pair_bit(i, j, N)) & 1) continue;
        if (c++ == q) { *pi = i; *pj = j; return; }
      }
  } else {
    q -= npk;
    for (int i = N - 2; i >= 0; i--)
      for (int j = N - 1; j > i; j--) {
        if ((kick >> pair_bit(i, j, N)) & 1) continue;
        if (c++ == q) { *pi = i; *pj = j; return; }
      }
  }
  *pi = 0;
  *pj = 1;
}

// kepler_driftij_gamma!'s Jacobian part for one pair from its capture; h2 is
// the drift's half step.
// With dh.p the derivative by h follows there.
template <bool DRIFT_FIRST>
__device__ __forceinline__ void pair_record_from_capture(const Rec& cap, int coff, double m_i, double m_j, double h2,
                                                         const Rec& rec, int roff, const Rec& dh) {
  double v[PCAP];
#pragma unroll
  for (int q = 0; q < PCAP; q++) v[q] = cap.get(coff + q);
  const double *x0 = v, *v0 = v + 3;
  KepParams P;
  P.gamma = v[6]; P.g2 = v[7]; P.g3 = v[8]; P.r0 = v[9]; P.r0inv = v[10]; P.rinv = v[PCAP_RINV]; P.beta = v[12]; P.eta = v[13];
  P.fm1 = v[14]; P.gmh = v[15]; P.dfdt = v[16]; P.dgdtm1 = v[17];
  P.k = GNEWT * (m_i + m_j);
  P.h = h2;
  KepDeriv D;
  double K[36], psi[6];
  if (dh.p) {
    double by_h[6];
    kep_derivatives<DRIFT_FIRST, true>(P, D);
    kep_by_h<DRIFT_FIRST>(P, D, x0, v0, by_h);
#pragma unroll
    for (int r = 0; r < 6; r++) dh.put(r, by_h[r]);
  } else {
    kep_derivatives<DRIFT_FIRST, false>(P, D);
  }
  kep_block<DRIFT_FIRST>(P, D, x0, v0, K, psi);
  const double mijinv = rcp_fast(m_i + m_j);
#pragma unroll
  for (int q = 0; q < 36; q++) rec.put(roff + q, K[q]);
  rec.put(roff + PREC_MI, m_i * mijinv);
  rec.put(roff + PREC_MJ, m_j * mijinv);
#pragma unroll
  for (int r = 0; r < 3; r++) {
    rec.put(roff + PREC_PSI + r, psi[r]);
    rec.put(roff + PREC_PSI + 3 + r, psi[3 + r]);
    rec.put(roff + PREC_B + r, mijinv * fma(P.fm1, x0[r], P.gmh * v0[r]));
    rec.put(roff + PREC_B + 3 + r, mijinv * fma(P.dfdt, x0[r], P.dgdtm1 * v0[r]));
  }
}

}  // namespace nbg
