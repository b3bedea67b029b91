// nbg_search.cuh -- transit searches of kick-free groups: findtransit!
// (src/transits/timing.jl:31-109) for a detection queued by the orbit producer.
//
// Newton iterations on partial AHL21 steps from the state at the detecting step's
// end, on x and v alone, with the physical time derivative of g
// (gdot_physical) where the reference builds the full gradient step to read g's
// step derivative: both reach the same root of g to rounding.  With grad the
// converged partial step's captures become pair records, dq/dt is carried
// forward through them and w^T S(dt0) backward (dtbvdq!, timing.jl:155-193); the
// corrector's Jacobian is applied pair by pair in both, never formed.
//
// Two forms, bitwise the same: one lane per search (many searches), and a
// block's lanes per search (orbit_lanes_kernel's layout) while few systems run
// and a search's latency counts.  Both are bound by the FP64 instructions one
// warp issues after another.  One lane -> a block's lanes, ms: 203 mixed systems
// over 80 steps 92 -> 47, one system over 400 steps of eight bodies 158 -> 148,
// over 203 of six with TransitParameters 56 -> 53.
#pragma once
#include "nbg_jacobian.cuh"
#include "nbg_orbit_team.cuh"

namespace nbg {

constexpr int SEARCH_ITMAX = 20;

// Sky-plane g and its physical time derivative from the two bodies'
// accelerations (timing.jl:141-144): |dv|^2 plus the relative acceleration.
template <int N>
__device__ __forceinline__ double gdot_from(const Sys<N>& s, int i, int j, const double* ai, const double* aj) {
  const double dvx = s.v[3 * j] - s.v[3 * i], dvy = s.v[3 * j + 1] - s.v[3 * i + 1];
  const double dx = s.x[3 * j] - s.x[3 * i], dy = s.x[3 * j + 1] - s.x[3 * i + 1];
  return dvx * dvx + dvy * dvy + dx * (aj[0] - ai[0]) + dy * (aj[1] - ai[1]);
}
// acceleration of body c by body b in the sky plane
template <int N>
__device__ __forceinline__ void sky_pull(const Sys<N>& s, int b, int c, double* f) {
  double d[3];
#pragma unroll
  for (int k = 0; k < 3; k++) d[k] = s.x[3 * b + k] - s.x[3 * c + k];
  const double r2 = norm2(d);
  const double w = GNEWT * s.m[b] / (r2 * sqrt(r2));
  f[0] = w * d[0];
  f[1] = w * d[1];
}
template <int N>
__device__ __forceinline__ double gdot_physical(const Sys<N>& s, int i, int j) {
  double ai[2] = {0.0, 0.0}, aj[2] = {0.0, 0.0}, f[2];
  for (int b = 0; b < N; b++) {
    if (b != i) {
      sky_pull(s, b, i, f);
      ai[0] += f[0];
      ai[1] += f[1];
    }
    if (b != j) {
      sky_pull(s, b, j, f);
      aj[0] += f[0];
      aj[1] += f[1];
    }
  }
  return gdot_from(s, i, j, ai, aj);
}

// ------------------------------------------------- the corrector, pair by pair
// dr, da: changes of r and of a_i - a_j; the notation is phi_columns'.

// change of the pair's acceleration term
__device__ __forceinline__ void accel_tangent(const double* r, double ri, const double* dr, double* t) {
  const double ri2 = ri * ri, f2 = (GNEWT * ri) * ri2, g5 = 3.0 * f2 * ri2;
  const double c = g5 * fma(r[2], dr[2], fma(r[1], dr[1], r[0] * dr[0]));
#pragma unroll
  for (int k = 0; k < 3; k++) t[k] = fma(f2, dr[k], -(c * r[k]));
}

struct CorrPair {
  double ri2, fac1, f3, fr, fac2, q3, gri;
};
__device__ __forceinline__ CorrPair corr_pair(const double* r, const double* a, double r2, double ri, double mij,
                                              double coeff) {
  CorrPair c;
  c.ri2 = ri * ri;
  c.fac1 = (coeff * ri) * (c.ri2 * c.ri2);
  c.f3 = 3.0 * c.fac1;
  c.fr = c.fac1 * r2;
  c.gri = (2.0 * GNEWT) * ri;
  c.fac2 = fma(c.gri, mij, 3.0 * fma(a[2], r[2], fma(a[1], r[1], a[0] * r[0])));
  c.q3 = c.gri * c.ri2 * mij;
  return c;
}

// change of F, plus `own` times F itself
__device__ __forceinline__ void corr_tangent(const double* r, const double* a, double r2, double ri, double mij,
                                             double coeff, const double* dr, const double* da, double own, double* f) {
  const CorrPair c = corr_pair(r, a, r2, ri, mij, coeff);
  const double rd = fma(r[2], dr[2], fma(r[1], dr[1], r[0] * dr[0]));
  const double along = fma(a[2], dr[2], fma(a[1], dr[1], a[0] * dr[0])) + fma(r[2], da[2], fma(r[1], da[1], r[0] * da[0]));
  const double diag = c.fac1 * c.fac2;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double F = c.fac1 * fma(r[k], c.fac2, -(r2 * a[k]));
    const double e = fma(-5.0 * c.ri2, F, -(c.fac1 * fma(c.q3, r[k], 2.0 * a[k])));
    f[k] = fma(own, F, fma(e, rd, fma(c.f3 * r[k], along, fma(diag, dr[k], -(c.fr * da[k])))));
  }
}

// From the adjoint velocities of i and j: the adjoints of r (er), of a_i - a_j
// (za) and of the two masses (pm).
__device__ __forceinline__ void corr_adjoint(const double* r, const double* a, double r2, double ri, double mi,
                                             double mj, double coeff, const double* ui, const double* uj, double* er,
                                             double* za, double* pm) {
  const CorrPair c = corr_pair(r, a, r2, ri, mi + mj, coeff);
  double w[3], fi = 0.0, fj = 0.0, ew = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) w[k] = fma(mj, ui[k], -(mi * uj[k]));
  const double rw = fma(r[2], w[2], fma(r[1], w[1], r[0] * w[0]));
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double F = c.fac1 * fma(r[k], c.fac2, -(r2 * a[k]));
    fi = fma(F, ui[k], fi);
    fj = fma(F, uj[k], fj);
    ew = fma(fma(-5.0 * c.ri2, F, -(c.fac1 * fma(c.q3, r[k], 2.0 * a[k]))), w[k], ew);
  }
  const double t = c.f3 * rw, diag = c.fac1 * c.fac2, g = (c.fac1 * c.gri) * rw;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    er[k] = fma(ew, r[k], fma(t, a[k], diag * w[k]));
    za[k] = fma(t, r[k], -(c.fr * w[k]));
  }
  pm[0] = g - fj;
  pm[1] = g + fi;
}

// From the adjoint accelerations of i and j: the adjoints of r and the masses.
__device__ __forceinline__ void accel_adjoint(const double* r, double ri, double mi, double mj, const double* ai,
                                              const double* aj, double* er, double* pm) {
  const double ri2 = ri * ri, f2 = (GNEWT * ri) * ri2, g5 = 3.0 * f2 * ri2;
  double y[3], pi = 0.0, pj = 0.0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    y[k] = fma(mi, aj[k], -(mj * ai[k]));
    pi = fma(r[k], aj[k], pi);
    pj = fma(r[k], ai[k], pj);
  }
  const double c = g5 * fma(r[2], y[2], fma(r[1], y[1], r[0] * y[0]));
#pragma unroll
  for (int k = 0; k < 3; k++) er[k] = fma(f2, y[k], -(c * r[k]));
  pm[0] = f2 * pi;
  pm[1] = -(f2 * pj);
}

// ------------------------------------------------------- scratch of one search
// Elements of a search's scratch (Rec with its stride): captures, snapshots,
// pair records each followed by d(delxv)/dh.
__host__ __device__ constexpr int search_slot() { return PREC + 6; }
template <int N>
struct SearchAt {
  static constexpr int P = N * (N - 1) / 2;
  static constexpr int cap = 0, xs = 2 * P * PCAP, rec = xs + 6 * N, end = rec + 2 * P * search_slot();
};

// Record of pair slot q from the captures of the converged step; a pair without
// mass repeats the record of the last one that had mass (zero without any).
template <int N>
__device__ __forceinline__ void search_record(const Rec& scr, const double* m, int slot, double h2) {
  constexpr int P = SearchAt<N>::P;
  const Rec cap{scr.p + (size_t)SearchAt<N>::cap * scr.stride, scr.stride};
  const Rec rec{scr.p + (size_t)(SearchAt<N>::rec + slot * search_slot()) * scr.stride, scr.stride};
  int q = slot;
  while (q >= 0 && cap.get(q * PCAP + PCAP_RINV) == 0.0) q--;
  if (q < 0) {
    for (int e = 0; e < search_slot(); e++) rec.put(e, 0.0);
    return;
  }
  int i, j;
  pair_of_slot<N>(q, P, 0, &i, &j);
  const Rec dh{rec.p + (size_t)PREC * scr.stride, scr.stride};
  if (q < P) pair_record_from_capture<true>(cap, q * PCAP, m[i], m[j], h2, rec, 0, dh);
  else pair_record_from_capture<false>(cap, q * PCAP, m[i], m[j], h2, rec, 0, dh);
}

// One lane: dq/dt of the step at dt0, q[6b + r], forward through the records.
template <int N>
__device__ void search_dq(const Rec& scr, const double* m, const double* v_start, const double* v_end, double h,
                          double* q) {
  using At = SearchAt<N>;
  const double h2 = 0.5 * h;
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) {
      q[6 * b + k] = 0.5 * v_start[3 * b + k];
      q[6 * b + 3 + k] = 0.0;
    }
  double last[12];
  for (int r = 0; r < 12; r++) last[r] = 0.0;
  auto pair = [&](int i, int j, int slot) {
    const int ro = At::rec + slot * search_slot();
    const bool stale = scr.get(At::cap + slot * PCAP + PCAP_RINV) == 0.0;
    const double mi = scr.get(ro + PREC_MI), mj = scr.get(ro + PREC_MJ);
    double d[6];
#pragma unroll
    for (int l = 0; l < 6; l++) d[l] = q[6 * i + l] - q[6 * j + l];
#pragma unroll
    for (int r = 0; r < 6; r++) {
      double u = stale ? 0.0 : 0.5 * scr.get(ro + PREC + r);
#pragma unroll
      for (int l = 0; l < 6; l++) u = fma(scr.get(ro + 6 * r + l), d[l], u);
      // a pair without mass keeps dqdt_ij, too, as the last pair left it (ahl21.jl:713)
      last[r] = fma(mj, u, stale ? fma(0.5, last[r], q[6 * i + r]) : q[6 * i + r]);
      last[6 + r] = fma(-mi, u, stale ? fma(0.5, last[6 + r], q[6 * j + r]) : q[6 * j + r]);
      q[6 * i + r] = last[r];
      q[6 * j + r] = last[6 + r];
    }
  };
  int slot = 0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) pair(i, j, slot++);
  double da[3 * N];
  for (int k = 0; k < 3 * N; k++) da[k] = 0.0;
  const double coeff = phis_coeff(h), hi3 = 3.0 / h;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      double r[3], dr[3], t[3];
      for (int k = 0; k < 3; k++) {
        r[k] = scr.get(At::xs + 3 * i + k) - scr.get(At::xs + 3 * j + k);
        dr[k] = q[6 * i + k] - q[6 * j + k];
      }
      accel_tangent(r, rsqrt_fast(norm2(r)), dr, t);
      for (int k = 0; k < 3; k++) {
        da[3 * i + k] = fma(-m[j], t[k], da[3 * i + k]);
        da[3 * j + k] = fma(m[i], t[k], da[3 * j + k]);
      }
    }
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      double r[3], a[3], dr[3], dij[3], f[3];
      for (int k = 0; k < 3; k++) {
        r[k] = scr.get(At::xs + 3 * i + k) - scr.get(At::xs + 3 * j + k);
        a[k] = scr.get(At::xs + 3 * N + 3 * i + k) - scr.get(At::xs + 3 * N + 3 * j + k);
        dr[k] = q[6 * i + k] - q[6 * j + k];
        dij[k] = da[3 * i + k] - da[3 * j + k];
      }
      const double r2 = norm2(r);
      corr_tangent(r, a, r2, rsqrt_fast(r2), m[i] + m[j], coeff, dr, dij, hi3, f);
      for (int k = 0; k < 3; k++) {
        q[6 * i + 3 + k] = fma(m[j], f[k], q[6 * i + 3 + k]);
        q[6 * j + 3 + k] = fma(-m[i], f[k], q[6 * j + 3 + k]);
      }
    }
  for (int i = N - 2; i >= 0; i--)
    for (int j = N - 1; j > i; j--) pair(i, j, slot++);
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++)
      q[6 * b + k] = q[6 * b + k] + fma(h2, q[6 * b + 3 + k], 0.5 * v_end[3 * b + k]);
}

// One lane: u <- S(dt0)^T u backward through the records, u[7b + r].
template <int N>
__device__ void search_adjoint(const Rec& scr, const double* m, double h, double* u) {
  using At = SearchAt<N>;
  const double h2 = 0.5 * h;
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) u[7 * b + 3 + k] = fma(h2, u[7 * b + k], u[7 * b + 3 + k]);
  int slot = 2 * At::P - 1;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) adj_pair(u, i, j, scr, At::rec + search_slot() * slot--);
  double za[3 * N];
  for (int k = 0; k < 3 * N; k++) za[k] = 0.0;
  const double coeff = phis_coeff(h);
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      double r[3], a[3], er[3], z[3], pm[2];
      for (int k = 0; k < 3; k++) {
        r[k] = scr.get(At::xs + 3 * i + k) - scr.get(At::xs + 3 * j + k);
        a[k] = scr.get(At::xs + 3 * N + 3 * i + k) - scr.get(At::xs + 3 * N + 3 * j + k);
      }
      const double r2 = norm2(r);
      corr_adjoint(r, a, r2, rsqrt_fast(r2), m[i], m[j], coeff, u + 7 * i + 3, u + 7 * j + 3, er, z, pm);
      for (int k = 0; k < 3; k++) {
        u[7 * i + k] = u[7 * i + k] + er[k];
        u[7 * j + k] = u[7 * j + k] - er[k];
        za[3 * i + k] = za[3 * i + k] + z[k];
        za[3 * j + k] = za[3 * j + k] - z[k];
      }
      u[7 * i + 6] = u[7 * i + 6] + pm[0];
      u[7 * j + 6] = u[7 * j + 6] + pm[1];
    }
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      double r[3], er[3], pm[2];
      for (int k = 0; k < 3; k++) r[k] = scr.get(At::xs + 3 * i + k) - scr.get(At::xs + 3 * j + k);
      accel_adjoint(r, rsqrt_fast(norm2(r)), m[i], m[j], za + 3 * i, za + 3 * j, er, pm);
      for (int k = 0; k < 3; k++) {
        u[7 * i + k] = u[7 * i + k] + er[k];
        u[7 * j + k] = u[7 * j + k] - er[k];
      }
      u[7 * i + 6] = u[7 * i + 6] + pm[0];
      u[7 * j + 6] = u[7 * j + 6] + pm[1];
    }
  for (int i = N - 2; i >= 0; i--)
    for (int j = N - 1; j > i; j--) adj_pair(u, i, j, scr, At::rec + search_slot() * slot--);
  for (int b = 0; b < N; b++)
    for (int k = 0; k < 3; k++) u[7 * b + 3 + k] = fma(h2, u[7 * b + k], u[7 * b + 3 + k]);
}

// The row w^T that starts adjoint r: of the transit time (dg), of v_sky's
// numerator, of b_sky^2 / 2 (timing.jl:155-191); entry e = 7b + component.
__device__ __forceinline__ double search_row(int r, int e, int ib, int ti, double dx, double dy, double dvx,
                                             double dvy) {
  const int b = e / 7, c = e % 7;
  if (b != ib && b != ti) return 0.0;
  double w = 0.0;
  if (r == 0) w = c == 0 ? dvx : c == 1 ? dvy : c == 3 ? dx : c == 4 ? dy : 0.0;
  if (r == 1) w = c == 3 ? dvx : c == 4 ? dvy : 0.0;
  if (r == 2) w = c == 0 ? dx : c == 1 ? dy : 0.0;
  return b == ib ? w : -w;
}

// What one thread writes of a finished search with grad beside the adjoint rows:
// gd, and for TransitParameters v_sky, dv_sky/dt and the two values.
// (q: dq/dt of the converged step, 6 a body.)
__device__ __forceinline__ void put_search(const GroupArgs& g, double* tr, double* ttout, int N, const double* q,
                                           int ib, int ti, double dx, double dy, double dvx, double dvy) {
  const int S = g.S;
  const double *qb = q + 6 * ib, *qt = q + 6 * ti;
  const double gd = fma(dvy, qb[1] - qt[1], fma(dvx, qb[0] - qt[0], fma(dy, qb[4] - qt[4], dx * (qb[3] - qt[3]))));
  if (!g.tbv) {
    tr[(size_t)(7 * N) * S] = gd;
    return;
  }
  const double vsky = sqrt(dvx * dvx + dvy * dvy);
  tr[(size_t)(21 * N) * S] = gd;
  tr[(size_t)(21 * N + 1) * S] = vsky;
  tr[(size_t)(21 * N + 2) * S] = fma(dvy, qb[4] - qt[4], dvx * (qb[3] - qt[3])) / vsky;
  ttout[1] = vsky;
  ttout[2] = dx * dx + dy * dy;
}

// A task of the queue.
struct SearchTask {
  int s, slot, c, ti, ib;
  double dt0, t;
};
template <int N>
__device__ __forceinline__ SearchTask search_task(const GroupArgs& g, int idx) {
  SearchTask k;
  const int* tk = g.task_i + 3 * idx;
  k.s = tk[0];
  k.slot = tk[1];
  k.c = tk[2];
  const int o = k.slot % (N - 1);
  k.ti = g.ti[k.s];
  k.ib = (o < k.ti) ? o : o + 1;
  const double* tf = g.task_f + (size_t)idx * (12 * N + 2);
  k.dt0 = tf[12 * N];
  k.t = tf[12 * N + 1];
  return k;
}

// ------------------------------------------------------------ one lane a search
template <int N>
__global__ void __launch_bounds__(TRANSIT_BS) transit_kernel(GroupArgs g, int chunk) {
  const int ntask = min(*g.task_count, g.task_cap);
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int G = gridDim.x * blockDim.x, S = g.S;
  const Rec none{nullptr, 0}, scr{g.grad ? g.tscratch + tid : nullptr, G};
  for (int idx = tid; idx < ntask; idx += G) {
    const SearchTask k = search_task<N>(g, idx);
    const double* tf = g.task_f + (size_t)idx * (12 * N + 2);
    Sys<N> wk;
    double a[3 * N], dt0 = k.dt0, stmp = 0.0, tt1 = dt0 + 1.0, tt2 = dt0 + 2.0;
    int iter = 0;
    for (int q = 0; q < N; q++) wk.m[q] = g.m[q * S + k.s];
    auto start = [&]() {
      for (int q = 0; q < 3 * N; q++) {
        wk.x[q] = tf[q];
        wk.v[q] = tf[3 * N + q];
        wk.xe[q] = tf[6 * N + q];
        wk.ve[q] = tf[9 * N + q];
      }
    };
    while (true) {
      tt2 = tt1;
      tt1 = dt0;
      start();
      plain_step<N>(wk, a, dt0, 0, none, none, none);
      const double gs = gsky(wk, k.ti, k.ib), gd = gdot_physical(wk, k.ti, k.ib);
      const double dt = -gs / gd;
      kahan(dt0, stmp, dt);
      iter += 1;
      if (iter >= SEARCH_ITMAX || dt0 == tt1 || dt0 == tt2) break;
    }
    if (iter >= SEARCH_ITMAX) atomicOr(g.status + k.s, NBG_STATUS_NEWTON_ITMAX);
    double* ttout = g.tt + g.off_tt[g.sysidx[k.s]] + (long long)(g.tbv ? 3 : 1) * (k.ib + (long long)N * k.c);
    if (g.grad) {
      start();
      plain_step<N>(wk, a, dt0, 0, scr, Rec{scr.p + (size_t)SearchAt<N>::xs * G, G}, none);
#pragma unroll 1
      for (int slot = 0; slot < 2 * SearchAt<N>::P; slot++) search_record<N>(scr, wk.m, slot, 0.5 * dt0);
      const double dvx = wk.v[3 * k.ib] - wk.v[3 * k.ti], dvy = wk.v[3 * k.ib + 1] - wk.v[3 * k.ti + 1];
      const double dx = wk.x[3 * k.ib] - wk.x[3 * k.ti], dy = wk.x[3 * k.ib + 1] - wk.x[3 * k.ti + 1];
      double q[7 * N];
      search_dq<N>(scr, wk.m, tf + 3 * N, wk.v, dt0, q);
      double* tr = g.trec + ((size_t)k.slot * trec_size(N, g.tbv)) * S + k.s;
      put_search(g, tr, ttout, N, q, k.ib, k.ti, dx, dy, dvx, dvy);
#pragma unroll 1
      for (int r = 0; r < (g.tbv ? 3 : 1); r++) {
        for (int e = 0; e < 7 * N; e++) q[e] = search_row(r, e, k.ib, k.ti, dx, dy, dvx, dvy);
        search_adjoint<N>(scr, wk.m, dt0, q);
        for (int e = 0; e < 7 * N; e++) tr[(size_t)(7 * N * r + e) * S] = q[e];
      }
      g.tflag[(size_t)k.slot * S + k.s] = k.c;
    } else if (g.tbv) {
      // TransitParameters without gradient (timing.jl:96-97): v_sky and
      // b_sky^2 of the last Newton iteration's state
      const double dvx = wk.v[3 * k.ib] - wk.v[3 * k.ti], dvy = wk.v[3 * k.ib + 1] - wk.v[3 * k.ti + 1];
      const double dx = wk.x[3 * k.ib] - wk.x[3 * k.ti], dy = wk.x[3 * k.ib + 1] - wk.x[3 * k.ti + 1];
      ttout[1] = sqrt(dvx * dvx + dvy * dvy);
      ttout[2] = dx * dx + dy * dy;
    }
    ttout[0] = k.t + dt0;
  }
}

// ------------------------------------------------------- a block's lanes a search
// orbit_lanes_kernel's layout (lanes_each(N) lanes per search): the partial steps
// are lanes_step; a lane per body forms the pulls of gdot_physical, a lane per
// pair slot its record and a lane per pair the corrector's terms, which each
// body's lanes add up in pair order; a pair's row of dq or u has a lane for each
// of its six entries.
template <int N>
struct SearchShared {
  LanesShared<N> l;
  Sys<N> st0;
  double scr[SearchAt<N>::end];
  double pull[2][N][2];
  double q[7 * N], z[3 * N];
  double f[N * (N - 1) / 2][8];
};

template <int N>
__device__ __forceinline__ void search_lanes_pair_dq(SearchShared<N>& sh, int i, int j, int slot, int t, double& last_i,
                                                     double& last_j) {
  const double* rc = sh.scr + SearchAt<N>::rec + slot * search_slot();
  const int l = t < 6 ? t : 0;
  double* q = sh.q;
  const double qi = q[6 * i + l], qj = q[6 * j + l];
  double d[6];
#pragma unroll
  for (int w = 0; w < 6; w++) d[w] = q[6 * i + w] - q[6 * j + w];
  const bool stale = sh.scr[SearchAt<N>::cap + slot * PCAP + PCAP_RINV] == 0.0;
  double u = stale ? 0.0 : 0.5 * rc[PREC + l];
#pragma unroll
  for (int w = 0; w < 6; w++) u = fma(rc[6 * l + w], d[w], u);
  last_i = fma(rc[PREC_MJ], u, stale ? fma(0.5, last_i, qi) : qi);
  last_j = fma(-rc[PREC_MI], u, stale ? fma(0.5, last_j, qj) : qj);
  __syncwarp();
  if (t < 6) {
    q[6 * i + l] = last_i;
    q[6 * j + l] = last_j;
  }
  __syncwarp();
}

// adj_pair on lanes 0-8: 0-5 the six entries, 6-8 the products with Psi and B
template <int N>
__device__ __forceinline__ void search_lanes_pair_adj(SearchShared<N>& sh, int i, int j, int slot, int t) {
  const double* rc = sh.scr + SearchAt<N>::rec + slot * search_slot();
  double* u = sh.q;
  const double mi = rc[PREC_MI], mj = rc[PREC_MJ];
  const int l = t < 6 ? t : 0;
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < 6; r++) {
    const double ui = u[7 * i + r], uj = u[7 * j + r];
    const double z = fma(mj, ui, -(mi * uj));
    const double x = t < 6 ? rc[6 * r + l] : t == 6 ? rc[PREC_PSI + r] : rc[PREC_B + r];
    acc = fma(x, t == 7 ? uj : t == 8 ? ui : z, acc);
  }
  const int base = threadIdx.x & 16;
  const double psi = __shfl_sync(0xffffffffu, acc, base + 6), bi = __shfl_sync(0xffffffffu, acc, base + 7),
               bj = __shfl_sync(0xffffffffu, acc, base + 8);
  if (t < 6) {
    u[7 * i + l] = u[7 * i + l] + acc;
    u[7 * j + l] = u[7 * j + l] - acc;
  } else if (t == 6) {
    u[7 * i + 6] = u[7 * i + 6] + (psi - bi);
    u[7 * j + 6] = u[7 * j + 6] + (psi + bj);
  }
  __syncwarp();
}

template <int N>
__global__ void __launch_bounds__(32 * lanes_warps(N)) transit_lanes_kernel(GroupArgs g, int chunk) {
  extern __shared__ double search_smem[];
  using At = SearchAt<N>;
  constexpr int T = lanes_each(N), P = At::P, SYS = lanes_systems(N);
  const int t = threadIdx.x % T, sub = threadIdx.x / T, S = g.S;
  SearchShared<N>& sh = reinterpret_cast<SearchShared<N>*>(search_smem)[sub];
  Sys<N>& wk = sh.l.st;
  const int ntask = min(*g.task_count, g.task_cap);
  const Rec none{nullptr, 0};
  for (int base = blockIdx.x * SYS; base < ntask; base += gridDim.x * SYS) {
    const bool has = base + sub < ntask;
    const int idx = has ? base + sub : base;  // a half warp without a search repeats the other's and writes nothing
    const SearchTask k = search_task<N>(g, idx);
    const double* tf = g.task_f + (size_t)idx * (12 * N + 2);
    if (t < 3 * N) {
      sh.st0.x[t] = tf[t];
      sh.st0.v[t] = tf[3 * N + t];
      sh.st0.xe[t] = tf[6 * N + t];
      sh.st0.ve[t] = tf[9 * N + t];
    }
    if (t < N) wk.m[t] = g.m[t * S + k.s];
    lanes_sync<N>();
    int pi = 0, pj = t + 1;  // pair t's bodies
    while (pj >= N && pi < N - 2) {
      pi++;
      pj += pi + 1 - N;
    }
    if (t < P) {
      const double mij = wk.m[pi] + wk.m[pj], inv = 1.0 / mij;
      sh.l.pk[t] = GNEWT * mij;
      sh.l.pmi[t] = wk.m[pi] * inv;
      sh.l.pmj[t] = wk.m[pj] * inv;
    }
    auto start = [&](bool run) {
      if (run && t < 3 * N) {
        wk.x[t] = sh.st0.x[t];
        wk.v[t] = sh.st0.v[t];
        wk.xe[t] = sh.st0.xe[t];
        wk.ve[t] = sh.st0.ve[t];
      }
      lanes_sync<N>();
    };
    double dt0 = k.dt0, stmp = 0.0, tt1 = dt0 + 1.0, tt2 = dt0 + 2.0;
    int iter = 0;
    bool active = true;
    // every search of the block steps until the last has converged
    while (SYS > 1 ? __any_sync(0xffffffffu, active) : active) {
      start(active);
      lanes_step<N, false>(sh.l, t, active, dt0, 0, none, none, none);
      if (t < N) {
        if (t != k.ti) sky_pull(wk, t, k.ti, sh.pull[0][t]);
        if (t != k.ib) sky_pull(wk, t, k.ib, sh.pull[1][t]);
      }
      lanes_sync<N>();
      if (active) {
        tt2 = tt1;
        tt1 = dt0;
        double ai[2] = {0.0, 0.0}, aj[2] = {0.0, 0.0};
        for (int b = 0; b < N; b++) {
          if (b != k.ti) {
            ai[0] += sh.pull[0][b][0];
            ai[1] += sh.pull[0][b][1];
          }
          if (b != k.ib) {
            aj[0] += sh.pull[1][b][0];
            aj[1] += sh.pull[1][b][1];
          }
        }
        const double gs = gsky(wk, k.ti, k.ib), gd = gdot_from(wk, k.ti, k.ib, ai, aj);
        const double dt = -gs / gd;
        kahan(dt0, stmp, dt);
        iter += 1;
        if (iter >= SEARCH_ITMAX || dt0 == tt1 || dt0 == tt2) active = false;
      }
      lanes_sync<N>();
    }
    if (has && t == 0 && iter >= SEARCH_ITMAX) atomicOr(g.status + k.s, NBG_STATUS_NEWTON_ITMAX);
    double* ttout = g.tt + g.off_tt[g.sysidx[k.s]] + (long long)(g.tbv ? 3 : 1) * (k.ib + (long long)N * k.c);
    if (g.grad) {
      start(true);
      lanes_step<N, false>(sh.l, t, true, dt0, 0, Rec{sh.scr + At::cap, 1}, Rec{sh.scr + At::xs, 1}, none);
      for (int slot = t; slot < 2 * P; slot += T) search_record<N>(Rec{sh.scr, 1}, wk.m, slot, 0.5 * dt0);
      const double h2 = 0.5 * dt0, coeff = phis_coeff(dt0);
      double r[3], a[3], r2 = 0.0, ri = 0.0;  // pair t at the corrector
      lanes_sync<N>();
      if (t < P) {
#pragma unroll
        for (int w = 0; w < 3; w++) {
          r[w] = sh.scr[At::xs + 3 * pi + w] - sh.scr[At::xs + 3 * pj + w];
          a[w] = sh.scr[At::xs + 3 * N + 3 * pi + w] - sh.scr[At::xs + 3 * N + 3 * pj + w];
        }
        r2 = norm2(r);
        ri = rsqrt_fast(r2);
      }
      const int b = t / 3, w3 = t % 3;  // coordinate lane
      auto pair_at = [&](int o) { return o < b ? pair_bit(o, b, N) : pair_bit(b, o, N); };
      // ---- dq/dt
      if (t < 3 * N) {
        sh.q[6 * b + w3] = 0.5 * sh.st0.v[t];
        sh.q[6 * b + 3 + w3] = 0.0;
      }
      lanes_sync<N>();
      double last_i = 0.0, last_j = 0.0;
      if (threadIdx.x < 32)
        for (int i = 0, slot = 0; i < N - 1; i++)
          for (int j = i + 1; j < N; j++) search_lanes_pair_dq<N>(sh, i, j, slot++, t, last_i, last_j);
      lanes_sync<N>();
      double dr[3];
      if (t < P) {
#pragma unroll
        for (int w = 0; w < 3; w++) dr[w] = sh.q[6 * pi + w] - sh.q[6 * pj + w];
        accel_tangent(r, ri, dr, sh.f[t]);
      }
      lanes_sync<N>();
      if (t < 3 * N) {
        double da = 0.0;
        for (int o = 0; o < N; o++)
          if (o != b) da = fma(o < b ? wk.m[o] : -wk.m[o], sh.f[pair_at(o)][w3], da);
        sh.z[t] = da;
      }
      lanes_sync<N>();
      if (t < P) {
        double da[3];
#pragma unroll
        for (int w = 0; w < 3; w++) da[w] = sh.z[3 * pi + w] - sh.z[3 * pj + w];
        corr_tangent(r, a, r2, ri, wk.m[pi] + wk.m[pj], coeff, dr, da, 3.0 / dt0, sh.f[t]);
      }
      lanes_sync<N>();
      if (t < 3 * N) {
        double v = sh.q[6 * b + 3 + w3];
        for (int o = 0; o < N; o++)
          if (o != b) v = fma(o < b ? -wk.m[o] : wk.m[o], sh.f[pair_at(o)][w3], v);
        sh.q[6 * b + 3 + w3] = v;
      }
      lanes_sync<N>();
      if (threadIdx.x < 32)
        for (int i = N - 2, slot = P; i >= 0; i--)
          for (int j = N - 1; j > i; j--) search_lanes_pair_dq<N>(sh, i, j, slot++, t, last_i, last_j);
      lanes_sync<N>();
      if (t < 3 * N) sh.q[6 * b + w3] = sh.q[6 * b + w3] + fma(h2, sh.q[6 * b + 3 + w3], 0.5 * wk.v[t]);
      lanes_sync<N>();
      const double dvx = wk.v[3 * k.ib] - wk.v[3 * k.ti], dvy = wk.v[3 * k.ib + 1] - wk.v[3 * k.ti + 1];
      const double dx = wk.x[3 * k.ib] - wk.x[3 * k.ti], dy = wk.x[3 * k.ib + 1] - wk.x[3 * k.ti + 1];
      double* tr = g.trec + ((size_t)k.slot * trec_size(N, g.tbv)) * S + k.s;
      if (has && t == 0) put_search(g, tr, ttout, N, sh.q, k.ib, k.ti, dx, dy, dvx, dvy);
      // ---- adjoint rows
#pragma unroll 1
      for (int row = 0; row < (g.tbv ? 3 : 1); row++) {
        lanes_sync<N>();
        for (int e = t; e < 7 * N; e += T) sh.q[e] = search_row(row, e, k.ib, k.ti, dx, dy, dvx, dvy);
        lanes_sync<N>();
        if (t < 3 * N) sh.q[7 * b + 3 + w3] = fma(h2, sh.q[7 * b + w3], sh.q[7 * b + 3 + w3]);
        lanes_sync<N>();
        if (threadIdx.x < 32)
          for (int i = 0, slot = 2 * P - 1; i < N - 1; i++)
            for (int j = i + 1; j < N; j++) search_lanes_pair_adj<N>(sh, i, j, slot--, t);
        lanes_sync<N>();
        if (t < P)  // er in 0-2, za in 3-5, the masses in 6-7
          corr_adjoint(r, a, r2, ri, wk.m[pi], wk.m[pj], coeff, sh.q + 7 * pi + 3, sh.q + 7 * pj + 3, sh.f[t],
                       sh.f[t] + 3, sh.f[t] + 6);
        lanes_sync<N>();
        auto gather = [&](bool accel) {
          if (t < 3 * N) {
            double x = sh.q[7 * b + w3], z = 0.0;
            for (int o = 0; o < N; o++)
              if (o != b) {
                const double* f = sh.f[pair_at(o)];
                x = o < b ? x - f[w3] : x + f[w3];
                if (accel) z = o < b ? z - f[3 + w3] : z + f[3 + w3];
              }
            sh.q[7 * b + w3] = x;
            if (accel) sh.z[t] = z;
          }
          if (t < N) {
            double mm = sh.q[7 * t + 6];
            for (int o = 0; o < N; o++)
              if (o != t) mm = mm + (o < t ? sh.f[pair_bit(o, t, N)][7] : sh.f[pair_bit(t, o, N)][6]);
            sh.q[7 * t + 6] = mm;
          }
          lanes_sync<N>();
        };
        gather(true);
        if (t < P)
          accel_adjoint(r, ri, wk.m[pi], wk.m[pj], sh.z + 3 * pi, sh.z + 3 * pj, sh.f[t], sh.f[t] + 6);
        lanes_sync<N>();
        gather(false);
        if (threadIdx.x < 32)
          for (int i = N - 2, slot = P - 1; i >= 0; i--)
            for (int j = N - 1; j > i; j--) search_lanes_pair_adj<N>(sh, i, j, slot--, t);
        lanes_sync<N>();
        if (t < 3 * N) sh.q[7 * b + 3 + w3] = fma(h2, sh.q[7 * b + w3], sh.q[7 * b + 3 + w3]);
        lanes_sync<N>();
        if (has)
          for (int e = t; e < 7 * N; e += T) tr[(size_t)(7 * N * row + e) * S] = sh.q[e];
      }
      if (has && t == 0) g.tflag[(size_t)k.slot * S + k.s] = k.c;
    } else if (g.tbv && has && t == 0) {
      const double dvx = wk.v[3 * k.ib] - wk.v[3 * k.ti], dvy = wk.v[3 * k.ib + 1] - wk.v[3 * k.ti + 1];
      const double dx = wk.x[3 * k.ib] - wk.x[3 * k.ti], dy = wk.x[3 * k.ib + 1] - wk.x[3 * k.ti + 1];
      ttout[1] = sqrt(dvx * dvx + dvy * dvy);
      ttout[2] = dx * dx + dy * dy;
    }
    if (has && t == 0) ttout[0] = k.t + dt0;
    lanes_sync<N>();
  }
}

}  // namespace nbg
