// nbg_jacobian.cuh -- the Jacobian consumer: one GPU lane owns one column of
// jac_step (and of jac_error) of one system and applies the operator stream
// the orbit producer's captures were turned into.
//
// Every update of ahl21! on jac_step (src/integrator/ahl21/ahl21.jl:5-95) has
// the form J <- J + A J followed by comp_sum_matrix!(J, J_err, A J)
// (src/utils.jl:36-46); columns of J never mix, so a column is a complete
// unit of work.  The consumer keeps the 6N non-mass rows of its column in
// shared memory ([row][lane], conflict-free); the mass rows of J are unit
// rows that no operator touches (the library checks this on entry).
//
// The pair update uses the structure of jac_ij (ahl21.jl:734-750): rows of
// body i are mj*K, -mj*K on (x,v)_i, (x,v)_j and rows of body j are -mi*K,
// mi*K, so jac_ij * [J_i; J_j] = [mj u; -mi u] with u = K (J_i - J_j), plus
// the two mass columns (PREC in nbg_layout.cuh): 36 products instead of 144
// for the dense 12x12 block; the product is rounded differently from a dense
// BLAS product, which the reference's BLAS leaves unspecified anyway.
#pragma once
#include "nbg_operators.cuh"

namespace nbg {

// The reference's folds and compensated row updates as it has them: what the
// tests hold against; the consumer's steps below normalise instead.
//
// Kahan fold with a zero addend (comp_sum_matrix! on a zero entry).
__device__ __forceinline__ void fold(double& s, double& e) {
  double t = s + e;
  e = (s - t) + e;
  s = t;
}

// Whether fold(s, e) changes s or e.  It leaves both bitwise unchanged exactly
// when s + e rounds to s (same bits), s is finite (else s - s is NaN) and e is
// not -0 ((s - s) + -0 is +0).  After a compensated add the pair is normally
// in that state: the add leaves in e the rounding error of s, which s + e
// rounds away.  The test costs one FP64 add against the fold's three; the
// rest is integer work.
__device__ __forceinline__ bool fold_changes(double s, double e) {
  const unsigned long long sb = __double_as_longlong(s), eb = __double_as_longlong(e);
  const unsigned long long tb = __double_as_longlong(s + e);
  return tb != sb || ((sb >> 52) & 0x7ffull) == 0x7ffull || eb == 0x8000000000000000ull;
}

// fold() on rows 6 b + R0 .. 6 b + R0 + NR - 1 of every body b.  The warp
// first tests its lanes' rows and runs the folds only if one of them would
// change a row, so the result is the folds' result bitwise (each lane skips
// only when no lane of its group, itself included, would change).
template <int N, int BS, int R0, int NR>
__device__ __forceinline__ void fold_rows(double* J, double* E) {
  bool change = false;
#pragma unroll 1
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int r = R0; r < R0 + NR; r++) change |= fold_changes(J[(6 * b + r) * BS], E[(6 * b + r) * BS]);
  if (!__any_sync(__activemask(), change)) return;
#pragma unroll 1
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int r = R0; r < R0 + NR; r++) fold(J[(6 * b + r) * BS], E[(6 * b + r) * BS]);
}

// J <- J + A J on all non-mass rows: velocity rows take the product P,
// position rows a zero addend.  Every row is summed on its own, so the
// position rows' folds may run first.
template <int N, int BS>
__device__ __forceinline__ void add_velocity_rows(double* J, double* E, const double* P) {
  fold_rows<N, BS, 0, 3>(J, E);
#pragma unroll 1
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int k = 0; k < 3; k++) kahan(J[(6 * b + 3 + k) * BS], E[(6 * b + 3 + k) * BS], P[3 * b + k]);
}
template <int N, int BS>
__device__ __forceinline__ void fold_all(double* J, double* E) {
  fold_rows<N, BS, 0, 6>(J, E);
}

// The step's updates with the Kahan pair (S, E) normalised less often: an update
// adds its increment to E in one FMA, J is S + E wherever it is read, and
// (S, E) <- (S + E, (S - (S + E)) + E) follows not after every update but where
// E holds a large increment: after the first drift (position rows), after the
// forward sweep's pairs with body 0 (velocity rows; the pairs between planets
// then add to a small E until the backward sweep's last pairs) and at the end
// of the step.  An addition to E rounds at the size of the increments in it, as
// the increment's own product does: against an extended-precision consumer of
// the same records, 2000 steps of two 8-body systems leave 2.3e-13 and 2.5e-13
// of jac_step where a Kahan sum at every update leaves 3.3e-13 and 2.5e-13.
// Per column and pair 66 FP64 instructions instead of 102, and no folds; per
// column-step at three bodies 600 instead of 864.  FP64 issue bounds the
// kernel: over 4096 three-body systems and 2000 steps its launches, one after
// another, went from 327 to 219 ms.
//
// The corrector's and the kicks' operators depend on position differences alone
// (the sum of their blocks over all bodies is zero), so they are applied to
// J_d - J_0.
//
// MASS: the column is a mass column (c % 7 == 6); the other columns, six of
// seven, share no warp with them and carry none of their terms.

__device__ __forceinline__ void normalise(double& s, double& e, double t) {  // t = s + e
  e = (s - t) + e;
  s = t;
}

template <int N, int BS, bool MASS>
__device__ __forceinline__ void pair_update(double* S, double* E, int c, int i, int j, const Rec& rec, int roff) {
  double K[36];
#pragma unroll
  for (int q = 0; q < 36; q++) K[q] = rec.get(roff + q);
  const double mi = rec.get(roff + PREC_MI), mj = rec.get(roff + PREC_MJ);
  const bool ci = MASS && c == 7 * i + 6, cj = MASS && c == 7 * j + 6;
  double U[6], B[6];
  if (MASS) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      U[q] = (ci || cj) ? rec.get(roff + PREC_PSI + q) : 0.0;
      B[q] = (ci || cj) ? rec.get(roff + PREC_B + q) : 0.0;
    }
  }
  double D[6];
#pragma unroll
  for (int l = 0; l < 6; l++)
    D[l] = (S[(6 * i + l) * BS] - S[(6 * j + l) * BS]) + (E[(6 * i + l) * BS] - E[(6 * j + l) * BS]);
#pragma unroll
  for (int r = 0; r < 6; r++) {
    double u = MASS ? fma(K[r * 6], D[0], U[r]) : K[r * 6] * D[0];
#pragma unroll
    for (int l = 1; l < 6; l++) u = fma(K[r * 6 + l], D[l], u);
    double ei = fma(mj, u, E[(6 * i + r) * BS]), ej = fma(-mi, u, E[(6 * j + r) * BS]);
    if (MASS) {
      ei = ei + (cj ? B[r] : 0.0);
      ej = ej - (ci ? B[r] : 0.0);
    }
    E[(6 * i + r) * BS] = ei;
    E[(6 * j + r) * BS] = ej;
  }
}

template <int N, int BS, bool MASS>
__device__ __forceinline__ void corrector_update(const double* S, double* E, int c, const Rec& rec, int roff) {
  double D[3 * N];  // D[3d + k]: position rows of body d less those of body 0
#pragma unroll
  for (int k = 0; k < 3; k++) D[k] = S[k * BS] + E[k * BS];
#pragma unroll
  for (int d = 1; d < N; d++)
#pragma unroll
    for (int k = 0; k < 3; k++) D[3 * d + k] = (S[(6 * d + k) * BS] + E[(6 * d + k) * BS]) - D[k];
  const int cm = c / 7;
#pragma unroll 1
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int rb = roff + (3 * b + k) * (4 * N);
      double acc = MASS ? fma(rec.get(rb + 4), D[3], rec.get(rb + 4 * cm + 3)) : rec.get(rb + 4) * D[3];
#pragma unroll
      for (int q = 1; q < 3 * (N - 1); q++) acc = fma(rec.get(rb + 4 + 4 * (q / 3) + q % 3), D[3 + q], acc);
      E[(6 * b + 3 + k) * BS] = E[(6 * b + 3 + k) * BS] + acc;
    }
}

// One recorded step on this column (ahl21.jl:5-95, the jac_step updates).  S and
// E arrive and leave normalised (S + E rounds to S).  The first kick's product is
// formed before the drift and counts after it (ahl21.jl:16-23): it goes to E of
// the velocity rows, whose S the drift reads.
template <int N, int BS, bool MASS, bool KICK>
__device__ __forceinline__ void column_step(double* S, double* E, int c, double h, uint64_t kick, const Rec& rec) {
  const double h2 = 0.5 * h;
  int roff = 0;
  if (KICK) {
    corrector_update<N, BS, MASS>(S, E, c, rec, roff);
    roff += op_size(N);
  }
#pragma unroll 2
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int r = (6 * b + k) * BS;
      double s = S[r], e = fma(h2, S[r + 3 * BS], E[r]);
      normalise(s, e, s + e);
      S[r] = s;
      E[r] = e;
    }
#pragma unroll 1
  for (int i = 0; i < N - 1; i++) {
#pragma unroll 1
    for (int j = i + 1; j < N; j++) {
      if (KICK && ((kick >> pair_bit(i, j, N)) & 1)) continue;
      pair_update<N, BS, MASS>(S, E, c, i, j, rec, roff);
      roff += PREC;
    }
    if (N > 2 && i == 0) {
#pragma unroll 3
      for (int q = 0; q < 3 * N; q++) {
        const int r = (6 * (q / 3) + 3 + q % 3) * BS;
        double s = S[r], e = E[r];
        normalise(s, e, s + e);
        S[r] = s;
        E[r] = e;
      }
    }
  }
  corrector_update<N, BS, MASS>(S, E, c, rec, roff);
  roff += op_size(N);
#pragma unroll 1
  for (int i = N - 2; i >= 0; i--)
#pragma unroll 1
    for (int j = N - 1; j > i; j--) {
      if (KICK && ((kick >> pair_bit(i, j, N)) & 1)) continue;
      pair_update<N, BS, MASS>(S, E, c, i, j, rec, roff);
      roff += PREC;
    }
#pragma unroll 2
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int r = (6 * b + k) * BS, rv = r + 3 * BS;
      double sv = S[rv], ev = E[rv];
      const double tv = sv + ev;
      normalise(sv, ev, tv);
      S[rv] = sv;
      E[rv] = ev;
      double s = S[r], e = fma(h2, tv, E[r]);
      normalise(s, e, s + e);
      S[r] = s;
      E[r] = e;
    }
  if (KICK) {
    corrector_update<N, BS, MASS>(S, E, c, rec, roff);
#pragma unroll 3
    for (int q = 0; q < 3 * N; q++) {
      const int r = (6 * (q / 3) + 3 + q % 3) * BS;
      double sv = S[r], ev = E[r];
      normalise(sv, ev, sv + ev);
      S[r] = sv;
      E[r] = ev;
    }
  }
}

}  // namespace nbg
