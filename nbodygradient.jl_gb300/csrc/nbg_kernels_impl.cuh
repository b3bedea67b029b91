// nbg_kernels_impl.cuh -- the per-body-count kernels of libnbg_cuda and their
// launchers.  Included only by nbg_inst.cu, which instantiates them for one
// body count N per translation unit (the units compile in parallel).
//
// Work decomposition, per chunk of K steps:
//   orbit_chunk_kernel<N>     one lane per system (nbg_orbit_team.cuh: a team, or a
//                             block's lanes): x, v, transit detection
//                             (src/transits/timing.jl:3-28); writes the pairs'
//                             captures, the snapshots and the search tasks
//   transit_kernel<N>         one lane per search (nbg_search.cuh: a block's lanes;
//                             transit_kick_kernel with kick pairs): tt and the
//                             per-transit adjoint rows (timing.jl:31-193)
//   operator_*_kernel<N>      captures and snapshots into the step's records
//   jacobian_chunk_kernel<N>  one lane per (system, column of jac_step), or
//   jacobian_rows_kernel<N>   six: apply the records, form dq/dt of the last
//                             step and each transit's dtdq0 entries
// Systems are grouped by (N, grad, kick pattern) so that every warp runs one
// control-flow path; within a group systems are sorted longest first.
#pragma once
#include <cuda_pipeline.h>

#include <algorithm>

#include "../../include/nbg.h"
#include "nbg_jacobian.cuh"
#include "nbg_search.cuh"

namespace nbg {

// Orbit producer for one chunk of K steps of one group (one lane per system).
template <int N, bool KICK>
__global__ void __launch_bounds__(PROD_BS * PROD_MAX_WARPS) orbit_chunk_kernel(GroupArgs g, int chunk) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane >= g.spw) return;
  const int s = (blockIdx.x * (blockDim.x / PROD_BS) + warp) * g.spw + lane;
  if (s >= g.S || g.sysidx[s] < 0) return;
  const int S = g.S;
  const long long nst = g.nsteps[s];
  const long long k0 = chunk_first_step(g, chunk, s);
  if (k0 >= nst || k0 < 0) return;  // done, or admitted for a later chunk
  Sys<N> st;
  double a[3 * N];
  for (int q = 0; q < 3 * N; q++) {
    st.x[q] = g.x[q * S + s];
    st.v[q] = g.v[q * S + s];
    st.xe[q] = g.xe[q * S + s];
    st.ve[q] = g.ve[q * S + s];
  }
  for (int q = 0; q < N; q++) st.m[q] = g.m[q * S + s];
  double gsave[N];
  long long count[N];
  for (int q = 0; q < N; q++) {
    gsave[q] = g.gsave[q * S + s];
    count[q] = g.count[q * S + s];
  }
  const double t0 = g.t0[s], h = g.h[s], hI = g.hI[s];
  const int ntt = g.ntt[s], ti = g.ti[s];
  const uint64_t kick = KICK ? g.kick : 0;
  for (int kk = 0; kk < g.K; kk++) {
    const long long istep = k0 + kk;
    if (istep >= nst) break;
    const double hs = step_length(g, s, istep, nst, h);
    if (g.trajxv) {
      double* rx = g.trajxv + ((size_t)s * g.K + kk) * 6 * N;
      for (int q = 0; q < 3 * N; q++) {
        rx[q] = st.x[q];
        rx[3 * N + q] = st.v[q];
      }
    }
    // x, v only; the operators are built from the captures by the operator kernels
    Rec cap{nullptr, 0}, xs{nullptr, 0};
    if (g.grad) {
      cap = Rec{g.pcap + (size_t)kk * 2 * g.npk * PCAP * S + s, S};
      xs = Rec{g.xsnap + (size_t)kk * snap_count(KICK) * 3 * N * S + s, S};
    }
    const Rec vs{g.grad && istep == nst - 1 ? g.vsnap + s : nullptr, S};
    plain_step<N>(st, a, hs, kick, cap, xs, vs);
    if (g.notransit) continue;
    const double t = t0 + (double)(istep + 1) * h;
    for (int o = 0; o < N - 1; o++) detect_transit<N>(g, st, s, kk, o, ti, ntt, hI, t, gsave, count);
  }
  for (int q = 0; q < 3 * N; q++) {
    g.x[q * S + s] = st.x[q];
    g.v[q * S + s] = st.v[q];
    g.xe[q * S + s] = st.xe[q];
    g.ve[q * S + s] = st.ve[q];
  }
  for (int q = 0; q < N; q++) {
    g.gsave[q * S + s] = gsave[q];
    g.count[q * S + s] = count[q];
  }
  // or-ed in: the transit searches and the consumer of the previous chunk may
  // be or-ing theirs meanwhile
  if (!state_finite<N>(st)) atomicOr(g.status + s, NBG_STATUS_NONFINITE);
}


// findtransit! (src/transits/timing.jl:31-109) in groups with kick pairs (the
// others: nbg_search.cuh), one lane per search: Newton iterations on partial AHL21 steps
// from the end-of-step state, then (grad) the partial step at the converged
// dt0 with its operator records and the adjoint row u^T = w^T S(dt0) that the
// Jacobian consumer turns into dtdq0 (dtbvdq! row 1, timing.jl:155-171).
// The iterations take x, v only and the physical time derivative of g
// (gdot_physical) where the reference builds the full gradient step to read
// g's step derivative: both iterations stop at the same root of g to
// rounding; the converged search's step keeps the reference's derivative,
// which dtdq0 divides by.
//
// Everything after the Newton iterations, for one search on one lane: st is
// the search's start state, wk the last iterate's state, dt0 the converged
// step; the operator records of the final partial step go to this lane's
// column `lane_id` of tscratch (lane_ids in 0..lanes-1).
template <int N>
__device__ void search_finish(const GroupArgs& g, int s, int slot, int c, int ib, int ti, const Sys<N>& st,
                              Sys<N>& wk, double dt0, double t, int iter, Work<N>& w, int lane_id, int lanes) {
  const int S = g.S;
  const uint64_t kick = g.kick;
  if (iter >= 20) atomicOr(g.status + s, NBG_STATUS_NEWTON_ITMAX);
  const int nr = g.tbv ? 3 : 1;
  double* ttout = g.tt + g.off_tt[g.sysidx[s]] + (long long)nr * (ib + (long long)N * c);
  if (g.tbv && !g.grad) {
    // TransitParameters without gradient (timing.jl:96-97): v_sky and
    // b_sky^2 of the last Newton iteration's state
    const double dvx = wk.v[3 * ib] - wk.v[3 * ti], dvy = wk.v[3 * ib + 1] - wk.v[3 * ti + 1];
    const double dx = wk.x[3 * ib] - wk.x[3 * ti], dy = wk.x[3 * ib + 1] - wk.x[3 * ti + 1];
    ttout[1] = sqrt(dvx * dvx + dvy * dvy);
    ttout[2] = dx * dx + dy * dy;
  }
  if (g.grad) {
    wk = st;
    Rec rec{g.tscratch + lane_id, lanes};
    ahl21_step<N>(wk, w, dt0, kick, rec);
    double u[7 * N];
    for (int q = 0; q < 7 * N; q++) u[q] = 0.0;
    const double dvx = wk.v[3 * ib] - wk.v[3 * ti], dvy = wk.v[3 * ib + 1] - wk.v[3 * ti + 1];
    const double dx = wk.x[3 * ib] - wk.x[3 * ti], dy = wk.x[3 * ib + 1] - wk.x[3 * ti + 1];
    u[7 * ib + 0] = dvx;
    u[7 * ti + 0] = -dvx;
    u[7 * ib + 1] = dvy;
    u[7 * ti + 1] = -dvy;
    u[7 * ib + 3] = dx;
    u[7 * ti + 3] = -dx;
    u[7 * ib + 4] = dy;
    u[7 * ti + 4] = -dy;
    adjoint_step<N>(u, dt0, kick, rec);
    const double gd = gdot(wk, ti, ib);
    double* tr = g.trec + ((size_t)slot * trec_size(N, g.tbv)) * S + s;
    for (int q = 0; q < 7 * N; q++) tr[(size_t)q * S] = u[q];
    if (g.tbv) {
      // dtbvdq! rows 2 and 3 (timing.jl:173-191): v_sky and b_sky^2 of the
      // converged state, dv_sky/dt, and the adjoint rows of their
      // numerators (d v_sky: the sky velocity difference on the velocity
      // rows; d b_sky^2 / 2: the sky position difference on the position rows)
      const double vsky = sqrt(dvx * dvx + dvy * dvy);
      const double bsky2 = dx * dx + dy * dy;
      const double* q = wk.dqdt;
      const double dvdt = (dvx * (q[7 * ib + 3] - q[7 * ti + 3]) + dvy * (q[7 * ib + 4] - q[7 * ti + 4])) / vsky;
      for (int r = 0; r < 2; r++) {
        for (int e = 0; e < 7 * N; e++) u[e] = 0.0;
        if (r == 0) {
          u[7 * ib + 3] = dvx;
          u[7 * ti + 3] = -dvx;
          u[7 * ib + 4] = dvy;
          u[7 * ti + 4] = -dvy;
        } else {
          u[7 * ib + 0] = dx;
          u[7 * ti + 0] = -dx;
          u[7 * ib + 1] = dy;
          u[7 * ti + 1] = -dy;
        }
        adjoint_step<N>(u, dt0, kick, rec);
        for (int e = 0; e < 7 * N; e++) tr[(size_t)(7 * N * (r + 1) + e) * S] = u[e];
      }
      tr[(size_t)(21 * N) * S] = gd;
      tr[(size_t)(21 * N + 1) * S] = vsky;
      tr[(size_t)(21 * N + 2) * S] = dvdt;
      ttout[1] = vsky;
      ttout[2] = bsky2;
    } else {
      tr[(size_t)(7 * N) * S] = gd;
    }
    g.tflag[(size_t)slot * S + s] = c;
  }
  ttout[0] = t + dt0;
}

template <int N>
__global__ void __launch_bounds__(TRANSIT_BS) transit_kick_kernel(GroupArgs g, int chunk) {
  const int ntask = min(*g.task_count, g.task_cap);
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int G = gridDim.x * blockDim.x;
  const int S = g.S;
  Work<N> w;
  for (int idx = tid; idx < ntask; idx += G) {
    const int* tk = g.task_i + 3 * idx;
    const int s = tk[0], slot = tk[1], c = tk[2];
    const int o = slot % (N - 1);
    const int ti = g.ti[s];
    const int ib = (o < ti) ? o : o + 1;
    const double* tf = g.task_f + (size_t)idx * (12 * N + 2);
    Sys<N> st;
    for (int q = 0; q < 3 * N; q++) {
      st.x[q] = tf[q];
      st.v[q] = tf[3 * N + q];
      st.xe[q] = tf[6 * N + q];
      st.ve[q] = tf[9 * N + q];
    }
    for (int q = 0; q < N; q++) st.m[q] = g.m[q * S + s];
    for (int q = 0; q < 7 * N; q++) st.dqdt[q] = 0.0;
    double dt0 = tf[12 * N];
    const double t = tf[12 * N + 1];
    const uint64_t kick = g.kick;
    double stmp = 0.0, tt1 = dt0 + 1.0, tt2 = dt0 + 2.0;
    int iter = 0;
    Sys<N> wk;
    while (true) {
      tt2 = tt1;
      tt1 = dt0;
      wk = st;
      plain_step<N>(wk, w.a, dt0, kick, Rec{nullptr, 0}, Rec{nullptr, 0}, Rec{nullptr, 0});
      const double gs = gsky(wk, ti, ib);
      const double gd = gdot_physical(wk, ti, ib);
      const double dt = -gs / gd;
      kahan(dt0, stmp, dt);
      iter += 1;
      if (iter >= 20 || dt0 == tt1 || dt0 == tt2) break;
    }
    search_finish<N>(g, s, slot, c, ib, ti, st, wk, dt0, t, iter, w, tid, G);
  }
}

// Kepler-pair records of one chunk: one lane per (step, pair slot, system),
// consecutive lanes = consecutive systems, so a warp shares its pair.
template <int N>
__global__ void __launch_bounds__(OPS_BS) operator_pair_kernel(GroupArgs g, int chunk) {
  const int S = g.S, np2 = 2 * g.npk;
  const long long L = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= (long long)g.K * np2 * S) return;
  const int s = (int)(L % S);
  const long long rest = L / S;
  const int slot = (int)(rest % np2), kk = (int)(rest / np2);
  if (g.sysidx[s] < 0) return;
  const long long istep = chunk_first_step(g, chunk, s) + kk;
  if (istep >= g.nsteps[s] || istep < 0) return;
  const uint64_t kick = g.kick;
  Rec cap{g.pcap + (size_t)kk * np2 * PCAP * S + s, S};
  Rec rec{g.steprec + (size_t)kk * g.R * S + s, S};
  const int roff = (kick ? op_size(N) : 0) + slot * PREC + (slot >= g.npk ? op_size(N) : 0);
  // A pair with G (m_i + m_j) == 0 keeps the jac_ij of the last pair of the
  // step that had mass (ahl21.jl:713 returns before refilling it); zero at the
  // start of the step (zero_out!, ahl21.jl:8).
  int q = slot;
  while (q >= 0 && cap.get(q * PCAP + PCAP_RINV) == 0.0) q--;
  if (q < 0) {
    for (int e = 0; e < PREC; e++) rec.put(roff + e, 0.0);
    return;
  }
  int i, j;
  pair_of_slot<N>(q, g.npk, kick, &i, &j);
  const double mi = g.m[i * S + s], mj = g.m[j * S + s];
  const double h2 = 0.5 * step_length(g, s, istep, g.nsteps[s], g.h[s]);
  Rec dh{nullptr, 0};
  if (q == slot && istep == g.nsteps[s] - 1) dh = Rec{g.dh + (size_t)slot * 6 * S + s, S};
  if (q < g.npk) pair_record_from_capture<true>(cap, q * PCAP, mi, mj, h2, rec, roff, dh);
  else pair_record_from_capture<false>(cap, q * PCAP, mi, mj, h2, rec, roff, dh);
}

// Corrector records of one chunk of a group without kick pairs: one lane per
// (step, body whose four columns it forms, system).
template <int N>
__global__ void __launch_bounds__(OPS_BS) operator_phi_kernel(GroupArgs g, int chunk) {
  const int S = g.S;
  const long long L = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= (long long)g.K * N * S) return;
  const int s = (int)(L % S);
  const long long rest = L / S;
  const int d = (int)(rest % N), kk = (int)(rest / N);
  if (g.sysidx[s] < 0) return;
  const long long istep = chunk_first_step(g, chunk, s) + kk;
  if (istep >= g.nsteps[s] || istep < 0) return;
  const double h = step_length(g, s, istep, g.nsteps[s], g.h[s]);
  Rec xs{g.xsnap + (size_t)kk * snap_count(false) * 3 * N * S + s, S};
  Rec rec{g.steprec + (size_t)kk * g.R * S + s, S};
  double x[3 * N], a[3 * N], m[N], acc[12 * N];
  for (int q = 0; q < 3 * N; q++) {
    x[q] = xs.get(q);
    a[q] = xs.get(3 * N + q);
  }
  for (int q = 0; q < N; q++) m[q] = g.m[q * S + s];
  for (int q = 0; q < 12 * N; q++) acc[q] = 0.0;
  // the consumer reads position columns of J_d - J_0 only, none of body 0's
  // (4096 three-body systems over 2000 steps: 551 -> 535 ms)
  if (d == 0) phi_columns<N, false>(x, a, m, h, 0, d, acc);
  else phi_columns<N>(x, a, m, h, 0, d, acc);
  const int off_phi = g.npk * PREC;
  for (int r = 0; r < 3 * N; r++)
    for (int p = d == 0 ? 3 : 0; p < 4; p++) rec.put(off_phi + r * (4 * N) + 4 * d + p, acc[4 * r + p]);
}

// Corrector and kick records of one chunk of a group with kick pairs: one lane
// per (step, system).
template <int N>
__global__ void __launch_bounds__(OPS_BS) operator_kick_kernel(GroupArgs g, int chunk) {
  const int S = g.S;
  const long long L = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= (long long)g.K * S) return;
  const int s = (int)(L % S), kk = (int)(L / S);
  if (g.sysidx[s] < 0) return;
  const long long istep = chunk_first_step(g, chunk, s) + kk;
  if (istep >= g.nsteps[s] || istep < 0) return;
  const uint64_t kick = g.kick;
  const double h = step_length(g, s, istep, g.nsteps[s], g.h[s]);
  Rec xs{g.xsnap + (size_t)kk * snap_count(true) * 3 * N * S + s, S};
  Rec rec{g.steprec + (size_t)kk * g.R * S + s, S};
  Sys<N> st;
  Work<N> w;
  for (int q = 0; q < N; q++) st.m[q] = g.m[q * S + s];
  for (int q = 0; q < 3 * N; q++) st.x[q] = xs.get(q), st.v[q] = st.xe[q] = st.ve[q] = 0.0;
  phic<N>(st, w, h, kick);
  phisalpha<N>(st, w.a, h, kick);
  phisalpha_operator<N>(st, w, h, kick);
  const int off_phi = op_size(N) + g.npk * PREC;
  put_op(rec, off_phi, w.op, op_size(N));
  const double h6 = h / 6.0;
  for (int q = 0; q < 3 * N; q++) st.x[q] = xs.get(3 * N + q);
  kickfast<N>(st, w, h6, kick);
  put_op(rec, 0, w.op, op_size(N));
  for (int q = 0; q < 3 * N; q++) st.x[q] = xs.get(6 * N + q);
  kickfast<N>(st, w, h6, kick);
  put_op(rec, off_phi + op_size(N) + g.npk * PREC, w.op, op_size(N));
}

// dtdq0 entry of column c for one transit (dtbvdq!, timing.jl:155-193) from the
// products of its adjoint rows with the column.
template <int N>
__device__ __forceinline__ void put_transit(const GroupArgs& g, int gsys, int ib, int flag, int ntt, int c,
                                            const double* acc, const double* tr) {
  const int S = g.S, cb = c / 7, ck = c % 7;  // column c is d/d q0[ck] of body cb
  const long long at = ib + (long long)N * (flag + (long long)ntt * (ck + 7LL * cb));
  if (!g.tbv) {
    g.dtdq0[g.off_dq[gsys] + at] = -acc[0] / tr[(size_t)(7 * N) * S];
    return;
  }
  const double gd = tr[(size_t)(21 * N) * S], vsky = tr[(size_t)(21 * N + 1) * S];
  const double dvdt = tr[(size_t)(21 * N + 2) * S];
  const double d1 = -acc[0] / gd;
  double* out = g.dtdq0 + g.off_dq[gsys] + 3 * at;
  out[0] = d1;
  out[1] = acc[1] / vsky + dvdt * d1;
  out[2] = 2.0 * acc[2];
}

// The entries of this column for the transits of step kk.
template <int N, int BS>
__device__ __forceinline__ void column_transits(const GroupArgs& g, int s, int c, int kk, int ti, int ntt, int gsys,
                                                const double* J, const double* E) {
  const int S = g.S, ck = c % 7;
  for (int o = 0; o < N - 1; o++) {
    const int flag = g.tflag[(size_t)(kk * (N - 1) + o) * S + s];
    if (flag < 0) continue;
    const double* tr = g.trec + ((size_t)(kk * (N - 1) + o) * trec_size(N, g.tbv)) * S + s;
    const int ib = (o < ti) ? o : o + 1;
    // the rows of a body in six sums, added in order (the lane form has a lane for each)
    double acc[3];
#pragma unroll 1
    for (int w = 0; w < (g.tbv ? 3 : 1); w++) {
      double part[6];
#pragma unroll
      for (int r = 0; r < 6; r++) part[r] = 0.0;
#pragma unroll 1
      for (int b = 0; b < N; b++)
#pragma unroll
        for (int r = 0; r < 6; r++) {
          const double ur = tr[(size_t)(7 * N * w + 7 * b + r) * S];
          part[r] = fma(ur, E[(6 * b + r) * BS], fma(ur, J[(6 * b + r) * BS], part[r]));
        }
      double sum = part[0];
#pragma unroll
      for (int r = 1; r < 6; r++) sum = sum + part[r];
      if (ck == 6) sum = sum + tr[(size_t)(7 * N * w + c) * S];  // unit mass row of this column
      acc[w] = sum;
    }
    put_transit<N>(g, gsys, ib, flag, ntt, c, acc, tr);
  }
}

// dq/dt of a system's last step (the State's dqdt; ahl21.jl:9-14, :20-24, :36-42
// and so on): one more column that the step's operators act on, with the drift
// velocities, the drifts' derivative by h and the corrector's and the kicks'
// dv/dt added on the way.  It is formed here, from the last step's record, and
// not by the producers: there it made the last step a one-lane gradient step
// (2.8 ms at eight bodies, 0.15 ms at two) and kept that step's working arrays
// on every producer's stack.  Six lanes per system, one for each row of a body,
// five systems a warp; sh: DQ_DOUBLES of the warp's own.
template <int N>
constexpr int DQ_DOUBLES = (15 * N + 6 * (N * (N - 1) / 2)) * 5;
template <int N, bool KICK>
__device__ void dq_columns(const GroupArgs& g, int chunk, int first, double* sh) {
  constexpr int P = N * (N - 1) / 2, C = 5;
  const int lane = threadIdx.x & 31, l = lane % 6, col = lane < 30 ? lane / 6 : 0, S = g.S;
  const int s = first + col;
  const uint64_t kick = KICK ? g.kick : 0;
  bool live = lane < 30 && s < S && g.grad && g.sysidx[s] >= 0;
  const long long nst = live ? g.nsteps[s] : 0, k0 = live ? chunk_first_step(g, chunk, s) : 0;
  live = live && k0 >= 0 && nst > k0 && nst <= k0 + g.K;
  if (!__any_sync(0xffffffffu, live)) return;
  const int kk = live ? (int)(nst - 1 - k0) : 0, at = live ? s : 0;
  const Rec rec{g.steprec + (size_t)kk * g.R * S + at, S}, dh{g.dh + at, S}, vs{g.vsnap + at, S};
  const Rec cap{g.pcap + (size_t)kk * 2 * g.npk * PCAP * S + at, S};
  const Rec xs{g.xsnap + (size_t)kk * snap_count(KICK) * 3 * N * S + at, S};
  const double h = live ? step_length(g, s, nst - 1, nst, g.h[s]) : 1.0, h2 = 0.5 * h;
  // Q: dq/dt [6b + r]; D: position differences; A: accelerations by Kepler and
  // by kicked pairs; F, G: a pair's force and correction
  double *Q = sh, *D = Q + 6 * N * C, *A = D + 3 * N * C, *F = A + 6 * N * C, *G = F + 3 * P * C;
  auto mass = [&](int b) { return g.m[b * S + s]; };
  auto pair_at = [](int o, int b) { return o < b ? pair_bit(o, b, N) : pair_bit(b, o, N); };
  auto is_kick = [&](int pb) { return KICK && ((kick >> pb) & 1); };
  // G r / r^3 of every pair at the positions of snapshot `snap`, in F
  auto forces = [&](int snap) {
    int p = 0;
    for (int i = 0; i < N - 1; i++)
      for (int j = i + 1; j < N; j++, p++) {
        if (p % 6 != l || !live) continue;
        double rij[3], f[3];
        for (int k = 0; k < 3; k++) rij[k] = xs.get(3 * N * snap + 3 * i + k) - xs.get(3 * N * snap + 3 * j + k);
        const double r2 = norm2(rij);
        phis_accel(rij, r2, sqrt(r2), f);
        for (int k = 0; k < 3; k++) F[(3 * p + k) * C + col] = f[k];
      }
    __syncwarp();
  };
  // a kick over h / 6: its dv/dt and, on dq/dt, its operator at roff (the first: dq/dt is zero)
  auto kick_rows = [&](int snap, int roff) {
    forces(snap);
    if (roff >= 0 && live && l < 3)
      for (int d = 1; d < N; d++) D[(3 * d + l) * C + col] = Q[(6 * d + l) * C + col] - Q[l * C + col];
    __syncwarp();
    if (live)
      for (int row = l; row < 3 * N; row += 6) {
        const int b = row / 3, k = row % 3;
        double acc = 0.0, op = 0.0;
        if (roff >= 0)
          for (int q = 0; q < 3 * (N - 1); q++)
            acc = fma(rec.get(roff + row * (4 * N) + 4 + 4 * (q / 3) + q % 3), D[(3 + q) * C + col], acc);
        for (int o = 0; o < N; o++)
          if (o != b && is_kick(pair_at(o, b))) op = fma(o < b ? mass(o) : -mass(o), F[(3 * pair_at(o, b) + k) * C + col], op);
        const int r = (6 * b + 3 + k) * C + col;
        Q[r] = Q[r] + fma(1.0 / 6.0, op, acc);
      }
    __syncwarp();
  };
  for (int b = 0; b < N; b++)
    if (live) Q[(6 * b + l) * C + col] = 0.0;
  int roff = 0;
  if (KICK) {
    kick_rows(1, -1);
    roff += op_size(N);
  }
  __syncwarp();
  for (int b = 0; b < N; b++)
    if (live && l < 3) Q[(6 * b + l) * C + col] = fma(h2, Q[(6 * b + 3 + l) * C + col], 0.5 * vs.get(3 * b + l));
  double last_i = 0.0, last_j = 0.0;
  auto pair = [&](int i, int j, int slot) {
    const int ai = (6 * i + l) * C + col, aj = (6 * j + l) * C + col;
    double ti = 0.0, tj = 0.0, K[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, mi = 0.0, mj = 0.0, by_h = 0.0;
    bool stale = false;
    if (live) {
#pragma unroll
      for (int q = 0; q < 6; q++) K[q] = rec.get(roff + 6 * l + q);
      mi = rec.get(roff + PREC_MI);
      mj = rec.get(roff + PREC_MJ);
      stale = cap.get(slot * PCAP + PCAP_RINV) == 0.0;
      if (!stale) by_h = dh.get(slot * 6 + l);
      ti = Q[ai];
      tj = Q[aj];
    }
    const double d = ti - tj;
    double u = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q++) u = fma(K[q], __shfl_sync(0xffffffffu, d, 6 * col + q), u);
    // a pair without mass keeps dqdt_ij, too, as the last pair left it (ahl21.jl:713)
    const double w = fma(0.5, by_h, u);
    last_i = fma(mj, w, stale ? fma(0.5, last_i, ti) : ti);
    last_j = fma(-mi, w, stale ? fma(0.5, last_j, tj) : tj);
    if (live) {
      Q[ai] = last_i;
      Q[aj] = last_j;
    }
  };
  int slot = 0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if (!is_kick(pair_bit(i, j, N))) {
        pair(i, j, slot++);
        roff += PREC;
      }
  __syncwarp();
  if (live && l < 3)
    for (int d = 1; d < N; d++) D[(3 * d + l) * C + col] = Q[(6 * d + l) * C + col] - Q[l * C + col];
  forces(0);
  if (live)
    for (int row = l; row < 3 * N; row += 6) {  // accelerations, as the producer sums them
      const int b = row / 3, k = row % 3;
      double a = 0.0, ac = 0.0;
      for (int o = 0; o < N; o++)
        if (o != b) {
          const double f = F[(3 * pair_at(o, b) + k) * C + col], m = o < b ? mass(o) : -mass(o);
          if (is_kick(pair_at(o, b))) ac = fma(m, f, ac);
          else a = fma(m, f, a);
        }
      A[row * C + col] = a;
      A[(3 * N + row) * C + col] = ac;
    }
  __syncwarp();
  if (live) {
    int p = 0;
    for (int i = 0; i < N - 1; i++)
      for (int j = i + 1; j < N; j++, p++) {
        if (p % 6 != l) continue;
        const double* a = A + (is_kick(p) ? 3 * N * C : 0) + col;
        double rij[3], aij[3], f[3];
        for (int k = 0; k < 3; k++) {
          rij[k] = xs.get(3 * i + k) - xs.get(3 * j + k);
          aij[k] = a[(3 * i + k) * C] - a[(3 * j + k) * C];
        }
        const double r2 = norm2(rij);
        phis_corr(rij, r2, sqrt(r2), aij, is_kick(p) ? 0.0 : mass(i) + mass(j),
                  is_kick(p) ? phic_coeff(h) : phis_coeff(h), f);
        for (int k = 0; k < 3; k++) G[(3 * p + k) * C + col] = f[k];
      }
  }
  __syncwarp();
  if (live) {
    const double hi3 = 3.0 / h;  // the corrections go with h^3, phic!'s kick with 2h / 3
    for (int row = l; row < 3 * N; row += 6) {
      const int b = row / 3, k = row % 3;
      double acc = 0.0, op = 0.0, kv = 0.0;
      for (int q = 0; q < 3 * (N - 1); q++)
        acc = fma(rec.get(roff + row * (4 * N) + 4 + 4 * (q / 3) + q % 3), D[(3 + q) * C + col], acc);
      for (int o = 0; o < N; o++)
        if (o != b) {
          const int at3 = (3 * pair_at(o, b) + k) * C + col;
          op = fma(o < b ? -mass(o) : mass(o), G[at3], op);
          if (is_kick(pair_at(o, b))) kv = fma(o < b ? mass(o) : -mass(o), F[at3], kv);
        }
      if (KICK) acc = fma(2.0 / 3.0, kv, acc);
      const int r = (6 * b + 3 + k) * C + col;
      Q[r] = Q[r] + fma(hi3, op, acc);
    }
  }
  __syncwarp();
  roff += op_size(N);
  for (int i = N - 2; i >= 0; i--)
    for (int j = N - 1; j > i; j--)
      if (!is_kick(pair_bit(i, j, N))) {
        pair(i, j, slot++);
        roff += PREC;
      }
  __syncwarp();
  if (live && l < 3)
    for (int b = 0; b < N; b++) {
      const int r = (6 * b + l) * C + col;
      Q[r] = Q[r] + fma(h2, Q[r + 3 * C], 0.5 * vs.get(3 * N + 3 * b + l));
    }
  __syncwarp();
  if (KICK) kick_rows(2, roff);
  if (live)
    for (int b = 0; b < N; b++) {
      g.dqdt[(7 * b + l) * S + s] = Q[(6 * b + l) * C + col];
      if (l == 0) g.dqdt[(7 * b + 6) * S + s] = 0.0;
    }
}

// Jacobian consumer for one chunk of K steps (one lane per column).  The mass
// columns have blocks of their own: the first `plain` blocks hold the other 6N
// columns of every system, the next ones, up to `all`, the N mass columns; the
// last ones form dq/dt.
template <int N, int BS, bool MASS, bool KICK>
__device__ __forceinline__ void consume_chunk(const GroupArgs& g, int chunk, int s, int c, double* smem) {
  constexpr int M = 7 * N, R6 = 6 * N;
  if (s >= g.S || g.sysidx[s] < 0) return;
  const int S = g.S;
  const long long nst = g.nsteps[s];
  const long long k0 = chunk_first_step(g, chunk, s);
  if (k0 >= nst || k0 < 0) return;  // done, or admitted for a later chunk
  double* J = smem + threadIdx.x;
  double* E = smem + R6 * BS + threadIdx.x;
  double* Jg = g.Jint + (size_t)s * R6 * M + c;
  double* Eg = g.Eint + (size_t)s * R6 * M + c;
  for (int r = 0; r < R6; r++) {
    double jv = Jg[(size_t)r * M], ev = Eg[(size_t)r * M];
    if (k0 == 0) fold(jv, ev);  // a caller's pair may not be normalised
    J[r * BS] = jv;
    E[r * BS] = ev;
  }
  const double h = g.h[s];
  const int ntt = g.ntt[s], ti = g.ti[s];
  const int gsys = g.sysidx[s];
  for (int kk = 0; kk < g.K; kk++) {
    const long long istep = k0 + kk;
    if (istep >= nst) break;
    Rec rec{g.steprec + (size_t)kk * g.R * S + s, S};
    if (g.trajJ) {  // column c of jac_step at the start of the step; mass rows are unit rows
      double* rj = g.trajJ + (((size_t)s * g.K + kk) * M + c) * M;
      for (int r = 0; r < M; r++) rj[r] = (r % 7 == 6) ? ((r == c) ? 1.0 : 0.0) : J[(6 * (r / 7) + r % 7) * BS];
    }
    const double hs = step_length(g, s, istep, nst, h);
    column_step<N, BS, MASS, KICK>(J, E, c, hs, KICK ? g.kick : 0, rec);
    if (!g.notransit) column_transits<N, BS>(g, s, c, kk, ti, ntt, gsys, J, E);
  }
  bool finite = true;
  for (int r = 0; r < R6; r++) {
    Jg[(size_t)r * M] = J[r * BS];
    Eg[(size_t)r * M] = E[r * BS];
    finite = finite && isfinite(J[r * BS]);
  }
  if (!finite) atomicOr(g.status + s, NBG_STATUS_NONFINITE);
}

// 168 registers a thread at most: three blocks of four warps fit an SM and leave
// room for a producer or search warp beside them.
template <int N, bool KICK>
__global__ void __launch_bounds__(cons_bs(N), 3 * 128 / cons_bs(N)) jacobian_chunk_kernel(GroupArgs g, int chunk, int plain, int all) {
  extern __shared__ double smem[];
  constexpr int BS = cons_bs(N);
  if ((int)blockIdx.x < plain) {
    const int f = blockIdx.x * BS + threadIdx.x, q = f % (6 * N);
    consume_chunk<N, BS, false, KICK>(g, chunk, f / (6 * N), 7 * (q / 6) + q % 6, smem);
  } else if ((int)blockIdx.x < all) {
    const int f = (blockIdx.x - plain) * BS + threadIdx.x;
    consume_chunk<N, BS, true, KICK>(g, chunk, f / N, 7 * (f % N) + 6, smem);
  } else {
    static_assert(DQ_DOUBLES<N> * (BS / 32) <= 2 * 6 * N * BS, "dq_columns' share of the columns' shared memory");
    const int w = (blockIdx.x - all) * (BS / 32) + threadIdx.x / 32;
    dq_columns<N, KICK>(g, chunk, 5 * w, smem + DQ_DOUBLES<N> * (threadIdx.x / 32));
  }
}

// Jacobian consumer for latency-bound chunks (the orbit producer's lanes form
// runs for them): six lanes per column of jac_step, one for each row of a body,
// five columns a warp, two warps a block.
//
// With few systems a column's lane is alone with its 64 cycles per FP64
// instruction, so a step takes as long as the column's instructions.  Here a
// pair costs 11 instead of 66 (three for D, six for its row of u, one for each
// body) and the corrector's 3N rows go round the six lanes; lanes exchange D
// by shuffles and the corrector's differences through shared memory.  The
// block copies the next step's record to shared memory while it applies this
// one (cp.async), so no trip to memory is waited out.  Per column the FP64 work
// is that of the one-lane form within a tenth, and every value is formed by the
// same operations in the same order: bitwise the same columns.
// One system alone, one lane a column -> six: 400 steps of eight bodies with
// transits 161 -> 148 ms, 2000 of three 193 -> 191 ms, 203 of six 57 -> 52 ms
// (its consumer 0.26 -> 0.044 ms a step at eight bodies, 0.030 -> 0.0065 at three).
constexpr int ROWS_COLS = 5, ROWS_WARPS = 2;
__host__ __device__ constexpr int rows_plain_warps(int N) { return (6 * N + ROWS_COLS - 1) / ROWS_COLS; }
__host__ __device__ constexpr int rows_warps(int N) { return rows_plain_warps(N) + (N + ROWS_COLS - 1) / ROWS_COLS; }
__host__ __device__ constexpr int rows_record(int N, bool kick) {  // at most
  return N * (N - 1) * PREC + (kick ? 3 : 1) * op_size(N);
}
__host__ __device__ constexpr int rows_blocks(int N) { return (rows_warps(N) + ROWS_WARPS - 1) / ROWS_WARPS; }
template <int N, bool KICK>
struct RowsShared {
  double rec[2][rows_record(N, KICK)];
  double S[ROWS_WARPS][6 * N * ROWS_COLS], E[ROWS_WARPS][6 * N * ROWS_COLS], D[ROWS_WARPS][3 * N * ROWS_COLS];
  int flag[2][N];
};

template <int N, bool MASS>
__device__ __forceinline__ void rows_pair(double* Sw, double* Ew, const double* rc, int i, int j, bool ci, bool cj,
                                          int l, int col, bool live) {
  const int ai = (6 * i + l) * ROWS_COLS + col, aj = (6 * j + l) * ROWS_COLS + col;
  const double ei = Ew[ai], ej = Ew[aj];
  const double d = (Sw[ai] - Sw[aj]) + (ei - ej);
  const double* K = rc + 6 * l;
  double u = 0.0;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const double D = __shfl_sync(0xffffffffu, d, 6 * col + q);
    if (q == 0) u = MASS ? fma(K[0], D, (ci || cj) ? rc[PREC_PSI + l] : 0.0) : K[0] * D;
    else u = fma(K[q], D, u);
  }
  double ni = fma(rc[PREC_MJ], u, ei), nj = fma(-rc[PREC_MI], u, ej);
  if (MASS) {
    const double B = rc[PREC_B + l];
    ni = ni + (cj ? B : 0.0);
    nj = nj - (ci ? B : 0.0);
  }
  if (live) {
    Ew[ai] = ni;
    Ew[aj] = nj;
  }
}

// corrector_update on the warp's columns: velocity rows of an operator that acts
// on position differences.
template <int N, bool MASS>
__device__ __forceinline__ void rows_operator(const double* Sw, double* Ew, double* Dw, const double* rc, int cm, int l,
                                              int col, bool live) {
  if (live && l < 3) {
    const double t0 = Sw[l * ROWS_COLS + col] + Ew[l * ROWS_COLS + col];
#pragma unroll
    for (int d = 1; d < N; d++) {
      const int r = (6 * d + l) * ROWS_COLS + col;
      Dw[(3 * d + l) * ROWS_COLS + col] = (Sw[r] + Ew[r]) - t0;
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int row = l; row < 3 * N; row += 6) {
    const double* rb = rc + row * (4 * N);
    const double* D = Dw + 3 * ROWS_COLS + col;
    double acc = MASS ? fma(rb[4], D[0], rb[4 * cm + 3]) : rb[4] * D[0];
#pragma unroll
    for (int q = 1; q < 3 * (N - 1); q++) acc = fma(rb[4 + 4 * (q / 3) + q % 3], D[q * ROWS_COLS], acc);
    const int r = (6 * (row / 3) + 3 + row % 3) * ROWS_COLS + col;
    if (live) Ew[r] = Ew[r] + acc;
  }
  __syncwarp();
}

// column_step on the warp's five columns.
template <int N, bool MASS, bool KICK>
__device__ __forceinline__ void rows_step(double* Sw, double* Ew, double* Dw, const double* rec, int c, double h,
                                          uint64_t kick, int l, int col, bool live) {
  const double h2 = 0.5 * h;
  const int cm = c / 7;
  const double* rc = rec;
  if (KICK) {
    rows_operator<N, MASS>(Sw, Ew, Dw, rc, cm, l, col, live);
    rc += op_size(N);
  }
  if (live && l < 3) {
#pragma unroll
    for (int b = 0; b < N; b++) {
      const int r = (6 * b + l) * ROWS_COLS + col;
      double s = Sw[r], e = fma(h2, Sw[r + 3 * ROWS_COLS], Ew[r]);
      normalise(s, e, s + e);
      Sw[r] = s;
      Ew[r] = e;
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int i = 0; i < N - 1; i++) {
#pragma unroll 1
    for (int j = i + 1; j < N; j++) {
      if (KICK && ((kick >> pair_bit(i, j, N)) & 1)) continue;
      rows_pair<N, MASS>(Sw, Ew, rc, i, j, cm == i, cm == j, l, col, live);
      rc += PREC;
    }
    if (N > 2 && i == 0 && live && l >= 3) {
#pragma unroll
      for (int b = 0; b < N; b++) {
        const int r = (6 * b + l) * ROWS_COLS + col;
        double s = Sw[r], e = Ew[r];
        normalise(s, e, s + e);
        Sw[r] = s;
        Ew[r] = e;
      }
    }
    __syncwarp();
  }
  rows_operator<N, MASS>(Sw, Ew, Dw, rc, cm, l, col, live);
  rc += op_size(N);
#pragma unroll 1
  for (int i = N - 2; i >= 0; i--)
#pragma unroll 1
    for (int j = N - 1; j > i; j--) {
      if (KICK && ((kick >> pair_bit(i, j, N)) & 1)) continue;
      rows_pair<N, MASS>(Sw, Ew, rc, i, j, cm == i, cm == j, l, col, live);
      rc += PREC;
    }
#pragma unroll
  for (int b = 0; b < N; b++) {
    const int r = (6 * b + l) * ROWS_COLS + col;
    double s = Sw[r], e = Ew[r], t = s + e;
    const double tv = __shfl_sync(0xffffffffu, t, 6 * col + (l < 3 ? l + 3 : l));
    if (l < 3) {
      e = fma(h2, tv, e);
      t = s + e;
    }
    normalise(s, e, t);
    if (live) {
      Sw[r] = s;
      Ew[r] = e;
    }
  }
  __syncwarp();
  if (KICK) {
    rows_operator<N, MASS>(Sw, Ew, Dw, rc, cm, l, col, live);
    if (live && l >= 3)
      for (int b = 0; b < N; b++) {
        const int r = (6 * b + l) * ROWS_COLS + col;
        double s = Sw[r], e = Ew[r];
        normalise(s, e, s + e);
        Sw[r] = s;
        Ew[r] = e;
      }
    __syncwarp();
  }
}

template <int N, bool KICK>
__global__ void __launch_bounds__(32 * ROWS_WARPS) jacobian_rows_kernel(GroupArgs g, int chunk) {
  extern __shared__ double smem[];
  RowsShared<N, KICK>& sh = *reinterpret_cast<RowsShared<N, KICK>*>(smem);
  constexpr int M = 7 * N, R6 = 6 * N;
  const int s = blockIdx.x, S = g.S, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((int)blockIdx.y == rows_blocks(N)) {  // the last row of blocks forms dq/dt
    dq_columns<N, KICK>(g, chunk, 5 * (ROWS_WARPS * s + warp), smem + DQ_DOUBLES<N> * warp);
    return;
  }
  if (s >= S || g.sysidx[s] < 0) return;
  const int R = KICK ? g.R : rows_record(N, false);  // a kick group's record is shorter by its kicked pairs
  const long long nst = g.nsteps[s], k0 = chunk_first_step(g, chunk, s);
  if (k0 >= nst || k0 < 0) return;  // done, or admitted for a later chunk
  const int nk = (int)(nst - k0 < g.K ? nst - k0 : g.K);
  // this lane's column: warps 0..rows_plain_warps-1 the columns that are not mass columns, then the mass columns
  const int wid = blockIdx.y * ROWS_WARPS + warp, pw = rows_plain_warps(N);
  const bool mass = wid >= pw;
  const int l = lane % 6, col = lane < 30 ? lane / 6 : 0;
  const int q = (mass ? wid - pw : wid) * ROWS_COLS + col;
  const bool live = lane < 30 && wid < rows_warps(N) && q < (mass ? N : 6 * N);
  const int c = !live ? 0 : mass ? 7 * q + 6 : 7 * (q / 6) + q % 6;
  double *Sw = sh.S[warp], *Ew = sh.E[warp], *Dw = sh.D[warp];
  double* Jg = g.Jint + (size_t)s * R6 * M + c;
  double* Eg = g.Eint + (size_t)s * R6 * M + c;
  if (lane < 30)
    for (int b = 0; b < N; b++) {
      const int r = 6 * b + l;
      double jv = live ? Jg[(size_t)r * M] : 0.0, ev = live ? Eg[(size_t)r * M] : 0.0;
      if (k0 == 0) fold(jv, ev);  // a caller's pair may not be normalised
      Sw[r * ROWS_COLS + col] = jv;
      Ew[r * ROWS_COLS + col] = ev;
    }
  auto fetch = [&](int kk) {
    const double* src = g.steprec + (size_t)kk * R * S + s;
    double* dst = sh.rec[kk & 1];
    for (int e = tid; e < R; e += 32 * ROWS_WARPS) __pipeline_memcpy_async(dst + e, src + (size_t)e * S, sizeof(double));
    if (!g.notransit && tid < N - 1)
      __pipeline_memcpy_async(&sh.flag[kk & 1][tid], g.tflag + (size_t)(kk * (N - 1) + tid) * S + s, sizeof(int));
    __pipeline_commit();
  };
  const double h = g.h[s];
  const int ntt = g.ntt[s], ti = g.ti[s], gsys = g.sysidx[s];
  fetch(0);
#pragma unroll 1
  for (int kk = 0; kk < nk; kk++) {
    if (kk + 1 < nk) fetch(kk + 1);
    else __pipeline_commit();
    __pipeline_wait_prior(1);
    __syncthreads();
    if (g.trajJ && live) {  // column c of jac_step at the start of the step; mass rows are unit rows
      double* rj = g.trajJ + (((size_t)s * g.K + kk) * M + c) * M;
      for (int b = 0; b < N; b++) {
        rj[7 * b + l] = Sw[(6 * b + l) * ROWS_COLS + col];
        if (l == 0) rj[7 * b + 6] = (7 * b + 6 == c) ? 1.0 : 0.0;
      }
    }
    const double hs = step_length(g, s, k0 + kk, nst, h);
    if (mass) rows_step<N, true, KICK>(Sw, Ew, Dw, sh.rec[kk & 1], c, hs, g.kick, l, col, live);
    else rows_step<N, false, KICK>(Sw, Ew, Dw, sh.rec[kk & 1], c, hs, g.kick, l, col, live);
    if (!g.notransit)
      for (int o = 0; o < N - 1; o++) {
        const int flag = sh.flag[kk & 1][o];
        if (flag < 0) continue;
        const double* tr = g.trec + ((size_t)(kk * (N - 1) + o) * trec_size(N, g.tbv)) * S + s;
        double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
        for (int w = 0; w < (g.tbv ? 3 : 1); w++) {
          double part = 0.0;
          for (int b = 0; b < N; b++) {
            const double ur = tr[(size_t)(7 * N * w + 7 * b + l) * S];
            const int r = (6 * b + l) * ROWS_COLS + col;
            part = fma(ur, Ew[r], fma(ur, Sw[r], part));
          }
          double sum = __shfl_sync(0xffffffffu, part, 6 * col);
#pragma unroll
          for (int r = 1; r < 6; r++) sum = sum + __shfl_sync(0xffffffffu, part, 6 * col + r);
          if (mass) sum = sum + tr[(size_t)(7 * N * w + c) * S];  // unit mass row of this column
          acc[w] = sum;
        }
        if (live && l == 0) put_transit<N>(g, gsys, (o < ti) ? o : o + 1, flag, ntt, c, acc, tr);
      }
    __syncthreads();  // the next fetch overwrites this step's record
  }
  if (live) {
    bool finite = true;
    for (int b = 0; b < N; b++) {
      const int r = 6 * b + l;
      const double jv = Sw[r * ROWS_COLS + col];
      Jg[(size_t)r * M] = jv;
      Eg[(size_t)r * M] = Ew[r * ROWS_COLS + col];
      finite = finite && isfinite(jv);
    }
    if (!finite) atomicOr(g.status + s, NBG_STATUS_NONFINITE);
  }
}

// gsave[i] = g!(i, ti, x, v) for every occultor (Transits.jl:146-149).
template <int N>
__global__ void seed_gsave_kernel(GroupArgs g) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.S || g.sysidx[s] < 0) return;
  const int S = g.S, ti = g.ti[s];
  for (int i = 0; i < N; i++) {
    if (i == ti) continue;
    const double dx = g.x[(3 * ti) * S + s] - g.x[(3 * i) * S + s];
    const double dy = g.x[(3 * ti + 1) * S + s] - g.x[(3 * i + 1) * S + s];
    const double dvx = g.v[(3 * ti) * S + s] - g.v[(3 * i) * S + s];
    const double dvy = g.v[(3 * ti + 1) * S + s] - g.v[(3 * i + 1) * S + s];
    g.gsave[i * S + s] = dx * dvx + dy * dvy;
  }
}

// Dynamic shared memory above the default 48 KB must be allowed per kernel.
template <class K>
inline void allow_smem(K kernel, int bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <int N, bool KICK>
void launch_lanes(const GroupArgs& g, int chunk, cudaStream_t st) {
  const int smem = std::max(lanes_systems(N) * (int)sizeof(LanesShared<N>), g.prod_smem);
  allow_smem(orbit_lanes_kernel<N, KICK>, smem);
  orbit_lanes_kernel<N, KICK>
      <<<(g.S + lanes_systems(N) - 1) / lanes_systems(N), 32 * lanes_warps(N), smem, st>>>(g, chunk);
}

template <int N>
int launch_orbit(const GroupArgs& g, int chunk, cudaStream_t st) {
  // Without a layout of the caller's (nbg_set_producer_layout) a full group's
  // one-lane warps go three to a block, four at two bodies: one warp alone needs
  // registers that three consumer blocks leave on no SM, and its block waits for
  // one of theirs to end; which sizes that hits depends on how the consumer's
  // last wave ends. One, two, three, four warps a block, ms, with derivatives:
  // N = 2 1024 steps 1300 systems 64.3, 64.5, 63.7, 67.0, 3000 81.4, 75.7, 70.6, 73.5,
  // 4096 85.0, 83.9, 103.3, 77.0; N = 3 256 steps 1024 52.4, 52.6, 51.3, 53.3,
  // 3100 64.9, 64.9, 63.3, 65.5, 512 steps 4096 144.2, 139.4, 140.2, 139.1;
  // N = 4 128 steps 1700 61.5, 61.3, 60.1, 61.8, 3000 74.9, 71.6, 71.3, 80.2.
  // Without derivatives there is no consumer, and one warp a block is the fastest.
  const int W = g.pwarps > 0 ? g.pwarps : (!g.team && g.grad && g.S >= 1024) ? (N == 2 ? 4 : 3) : 1;
  if (g.wide) {
    if (g.kick) launch_lanes<N, true>(g, chunk, st);
    else launch_lanes<N, false>(g, chunk, st);
    return 0;
  }
  if (g.team && !g.kick) {
    constexpr int T = PROD_BS / team_lanes(N);
    const int smem = std::max(team_smem_bytes<N>(W), g.prod_smem);
    allow_smem(orbit_team_kernel<N>, smem);
    orbit_team_kernel<N><<<(g.S + W * T - 1) / (W * T), PROD_BS * W, smem, st>>>(g, chunk);
    return 0;
  }
  const int blocks = (g.S + W * g.spw - 1) / (W * g.spw);
  if (g.kick) {
    allow_smem(orbit_chunk_kernel<N, true>, g.prod_smem);
    orbit_chunk_kernel<N, true><<<blocks, PROD_BS * W, g.prod_smem, st>>>(g, chunk);
  } else {
    allow_smem(orbit_chunk_kernel<N, false>, g.prod_smem);
    orbit_chunk_kernel<N, false><<<blocks, PROD_BS * W, g.prod_smem, st>>>(g, chunk);
  }
  return 0;
}

template <int N, bool KICK>
void launch_consumer(const GroupArgs& g, int chunk, cudaStream_t st) {
  // the attributes are set per call: they belong to the current device
  if (g.rows) {
    // as every consumer block: none fits beside a tail producer's
    const int bytes = std::max((int)sizeof(RowsShared<N, KICK>), 24 * 1024);
    static_assert(sizeof(double) * DQ_DOUBLES<N> * ROWS_WARPS <= std::max<size_t>(sizeof(RowsShared<N, KICK>), 24 * 1024),
                  "dq_columns fits");
    allow_smem(jacobian_rows_kernel<N, KICK>, bytes);
    const dim3 grid(g.S, rows_blocks(N) + 1);
    jacobian_rows_kernel<N, KICK><<<grid, 32 * ROWS_WARPS, bytes, st>>>(g, chunk);
    return;
  }
  constexpr int BS = cons_bs(N);
  const int smem = 2 * 6 * N * BS * (int)sizeof(double);
  auto blocks = [](long long columns) { return (int)((columns + BS - 1) / BS); };
  const int plain = blocks((long long)g.S * 6 * N), all = plain + blocks((long long)g.S * N);
  const int dq = (g.S + 5 * (BS / 32) - 1) / (5 * (BS / 32));
  allow_smem(jacobian_chunk_kernel<N, KICK>, smem);
  jacobian_chunk_kernel<N, KICK><<<all + dq, BS, smem, st>>>(g, chunk, plain, all);
}

template <int N>
int launch_jac(const GroupArgs& g, int chunk, cudaStream_t st) {
  if (g.kick) launch_consumer<N, true>(g, chunk, st);
  else launch_consumer<N, false>(g, chunk, st);
  return 0;
}

template <int N>
int launch_transit(const GroupArgs& g, int chunk, cudaStream_t st) {
  if (g.kick) {
    allow_smem(transit_kick_kernel<N>, g.guard_smem);
    transit_kick_kernel<N><<<g.tgrid / TRANSIT_BS, TRANSIT_BS, g.guard_smem, st>>>(g, chunk);
  } else if (g.search_lanes) {
    const int smem = std::max(lanes_systems(N) * (int)sizeof(SearchShared<N>), g.guard_smem);
    allow_smem(transit_lanes_kernel<N>, smem);
    transit_lanes_kernel<N><<<g.tgrid / TRANSIT_BS, 32 * lanes_warps(N), smem, st>>>(g, chunk);
  } else {
    // An SM that runs blocks without shared memory gives it to L1, and a team or
    // lanes producer's block waits until that SM idles: the next chunk's then crowd
    // on a few.  Where no consumer block (24 KB or more) sees to it, the searches
    // ask for some themselves, 12 blocks an SM as its registers allow 8.  Without ->
    // with, no derivatives, 128 steps, ms: 2048 systems of five bodies 122 -> 64,
    // 1024 of six 143 -> 79, of eight 213 -> 118; one-lane producers are level
    // (2048 of four 50.0).
    const int smem = g.grad ? g.guard_smem : std::max(g.guard_smem, 18 * 1024);
    allow_smem(transit_kernel<N>, smem);
    transit_kernel<N><<<g.tgrid / TRANSIT_BS, TRANSIT_BS, smem, st>>>(g, chunk);
  }
  return 0;
}

template <int N>
int launch_operators(const GroupArgs& g, int chunk, cudaStream_t st) {
  long long lanes = (long long)g.K * 2 * g.npk * g.S;
  allow_smem(operator_pair_kernel<N>, g.guard_smem);
  if (lanes > 0)
    operator_pair_kernel<N><<<(unsigned)((lanes + OPS_BS - 1) / OPS_BS), OPS_BS, g.guard_smem, st>>>(g, chunk);
  if (g.kick) {
    lanes = (long long)g.K * g.S;
    allow_smem(operator_kick_kernel<N>, g.guard_smem);
    operator_kick_kernel<N><<<(unsigned)((lanes + OPS_BS - 1) / OPS_BS), OPS_BS, g.guard_smem, st>>>(g, chunk);
  } else {
    lanes = (long long)g.K * N * g.S;
    allow_smem(operator_phi_kernel<N>, g.guard_smem);
    operator_phi_kernel<N><<<(unsigned)((lanes + OPS_BS - 1) / OPS_BS), OPS_BS, g.guard_smem, st>>>(g, chunk);
  }
  return 0;
}

template <int N>
int launch_seed(const GroupArgs& g, cudaStream_t st) {
  int b = (g.S + 127) / 128;
  seed_gsave_kernel<N><<<b, 128, 0, st>>>(g);
  return 0;
}

}  // namespace nbg
