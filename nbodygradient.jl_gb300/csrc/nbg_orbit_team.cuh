// nbg_orbit_team.cuh -- the orbit producer with a team of lanes per system.
//
// The Kepler sweeps of an AHL21 step (ahl21.jl:25-27 forward, :56-58
// backward) update bodies i and j of each pair in a fixed order.  A pair's
// update reads and writes only x, v (and their Kahan errors) of its two
// bodies, so two pairs with no body in common commute exactly.  In the
// forward order (i = 0..N-2, j = i+1..N-1), the pairs that touch body b come
// in order of increasing i + j: (0,b), (1,b), ..., (b-1,b), (b,b+1), ...,
// (b,N-1).  The pairs with one value of i + j share no body.  Running the
// sweep "level by level" in increasing i + j, with the pairs of one level
// in parallel, therefore applies to every body the same updates in the same
// order as the sequential sweep: the result is bitwise identical.  The
// backward sweep is the exact reverse sequence, so it runs the levels in
// decreasing i + j.  phisalpha!'s two pair loops (the acceleration sums and
// the velocity kicks, ahl21.jl:558-700 without the gradient) follow the same
// pair order and run level by level too.
//
// A level holds at most floor(N/2) pairs, so a team of L = max(1, N/2) lanes
// runs one system, 32 / L systems per warp, the system's x, v, errors and
// masses in shared memory.  The critical path of a sweep drops from
// N(N-1)/2 to 2N-3 pair solves (N = 10: 45 -> 17; N = 8: 28 -> 13).
//
// Groups with kick pairs (pair[i,j] == true) take one lane or the lanes form.
#pragma once
#include "nbg_orbit.cuh"

namespace nbg {

__host__ __device__ constexpr int team_lanes(int N) { return N / 2 > 1 ? N / 2 : 1; }

// The pair of level `lev` (i + j == lev) that lane t of a team takes, if any.
template <int N>
__device__ __forceinline__ bool level_pair(int lev, int t, int* i, int* j) {
  const int imin = lev - (N - 1) > 0 ? lev - (N - 1) : 0;
  const int ii = imin + t;
  if (2 * ii >= lev) return false;  // i < j = lev - i
  *i = ii;
  *j = lev - ii;
  return true;
}

// One AHL21 step without gradient operators for a group with no kick pairs
// (ahl21_no_grad.jl:6-18 order), run by the L lanes of a team; `run` is
// false for lanes whose system does not step (they still meet every
// __syncwarp).  cap / xs as in ahl21_step.  a: the team's 3N acceleration
// scratch.
template <int N>
__device__ __forceinline__ void team_step(Sys<N>& s, double* a, int t, bool run, double h,
                                          const Rec& cap, const Rec& xs, const Rec& vs) {
  constexpr int L = team_lanes(N);
  constexpr int P = N * (N - 1) / 2;
  const double h2 = 0.5 * h;
  if (run)
    for (int q = t; q < 3 * N; q += L) {
      if (vs.p) vs.put(q, s.v[q]);
      kahan_fma(s.x[q], s.xe[q], h2, s.v[q]);
    }
  __syncwarp();
  for (int lev = 1; lev <= 2 * N - 3; lev++) {
    int i, j;
    if (run && level_pair<N>(lev, t, &i, &j))
      kepler_pair<N, true>(s, i, j, h2, cap, pair_bit(i, j, N) * PCAP);
    __syncwarp();
  }
  if (run) {
    if (xs.p)
      for (int q = t; q < 3 * N; q += L) xs.put(q, s.x[q]);
    for (int q = t; q < 3 * N; q += L) a[q] = 0.0;
  }
  __syncwarp();
  const double coeff = phis_coeff(h);
  for (int lev = 1; lev <= 2 * N - 3; lev++) {
    int i, j;
    if (run && level_pair<N>(lev, t, &i, &j)) phis_accel_pair<N>(s, a, i, j);
    __syncwarp();
  }
  if (run && xs.p)
    for (int q = t; q < 3 * N; q += L) xs.put(3 * N + q, a[q]);
  for (int lev = 1; lev <= 2 * N - 3; lev++) {
    int i, j;
    if (run && level_pair<N>(lev, t, &i, &j)) phis_kick_pair<N>(s, a, i, j, s.m[i] + s.m[j], coeff);
    __syncwarp();
  }
  for (int lev = 2 * N - 3; lev >= 1; lev--) {
    int i, j;
    if (run && level_pair<N>(lev, t, &i, &j))
      kepler_pair<N, false>(s, i, j, h2, cap, (P + (P - 1 - pair_bit(i, j, N))) * PCAP);
    __syncwarp();
  }
  if (run)
    for (int q = t; q < 3 * N; q += L) {
      if (vs.p) vs.put(3 * N + q, s.v[q]);
      kahan_fma(s.x[q], s.xe[q], h2, s.v[q]);
    }
  __syncwarp();
}

// Dynamic shared memory the team producer needs for W warps per block:
// per team a Sys<N>, 3N accelerations, N g values and N transit counts.
template <int N>
__host__ __device__ constexpr int team_smem_bytes(int W) {
  return W * (PROD_BS / team_lanes(N)) *
         (int)(sizeof(Sys<N>) + (3 * N + N) * sizeof(double) + N * sizeof(long long));
}

// Orbit producer, team form: L = team_lanes(N) lanes per system, T = 32 / L
// systems per warp (lanes beyond T * L idle), pwarps independent warps per
// block.  Same inputs, outputs and arithmetic as orbit_chunk_kernel<N> for
// groups without kick pairs.
template <int N>
__global__ void __launch_bounds__(PROD_BS * PROD_MAX_WARPS) orbit_team_kernel(GroupArgs g, int chunk) {
  constexpr int L = team_lanes(N);
  constexpr int T = PROD_BS / L;
  const int W = blockDim.x / PROD_BS;
  extern __shared__ double team_smem[];
  Sys<N>* sys = reinterpret_cast<Sys<N>*>(team_smem);
  double(*acc)[3 * N] = reinterpret_cast<double(*)[3 * N]>(sys + W * T);
  double(*gsv)[N] = reinterpret_cast<double(*)[N]>(acc + W * T);
  long long(*cnt)[N] = reinterpret_cast<long long(*)[N]>(gsv + W * T);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int team = lane / L, t = lane % L;
  const bool in_team = team < T;
  const int tm = warp * T + (in_team ? team : 0);  // idle lanes alias their warp's team 0 but never write
  const int s = blockIdx.x * W * T + tm;
  const int S = g.S;
  bool valid = in_team && s < S && g.sysidx[s] >= 0;
  const long long nst = valid ? g.nsteps[s] : 0;
  const long long k0 = valid ? chunk_first_step(g, chunk, s) : 0;
  if (k0 >= nst || k0 < 0) valid = false;  // done, or admitted for a later chunk
  Sys<N>& st = sys[tm];
  if (valid) {
    for (int q = t; q < 3 * N; q += L) {
      st.x[q] = g.x[q * S + s];
      st.v[q] = g.v[q * S + s];
      st.xe[q] = g.xe[q * S + s];
      st.ve[q] = g.ve[q * S + s];
    }
    for (int q = t; q < N; q += L) {
      st.m[q] = g.m[q * S + s];
      gsv[tm][q] = g.gsave[q * S + s];
      cnt[tm][q] = g.count[q * S + s];
    }
  }
  __syncwarp();
  const double t0 = valid ? g.t0[s] : 0.0, h = valid ? g.h[s] : 0.0, hI = valid ? g.hI[s] : 0.0;
  const int ntt = valid ? g.ntt[s] : 0, ti = valid ? g.ti[s] : 0;
  for (int kk = 0; kk < g.K; kk++) {
    const long long istep = k0 + kk;
    const bool run = valid && istep < nst;
    if (!__any_sync(0xffffffffu, run)) break;
    Rec cap{nullptr, 0}, xs{nullptr, 0};
    if (g.grad) {
      cap = Rec{g.pcap + (size_t)kk * 2 * g.npk * PCAP * S + s, S};
      xs = Rec{g.xsnap + (size_t)kk * snap_count(false) * 3 * N * S + s, S};
    }
    const double hs = run ? step_length(g, s, istep, nst, h) : h;
    if (run && g.trajxv) {
      double* rx = g.trajxv + ((size_t)s * g.K + kk) * 6 * N;
      for (int q = t; q < 3 * N; q += L) {
        rx[q] = st.x[q];
        rx[3 * N + q] = st.v[q];
      }
    }
    const Rec vs{run && g.grad && istep == nst - 1 ? g.vsnap + s : nullptr, S};
    team_step<N>(st, acc[tm], t, run, hs, cap, xs, vs);
    // occultor o on lane o % L
    if (run && !g.notransit)
      for (int o = t; o < N - 1; o += L)
        detect_transit<N>(g, st, s, kk, o, ti, ntt, hI, t0 + (double)(istep + 1) * h, &gsv[tm][0], &cnt[tm][0]);
    __syncwarp();
  }
  if (valid) {
    for (int q = t; q < 3 * N; q += L) {
      g.x[q * S + s] = st.x[q];
      g.v[q * S + s] = st.v[q];
      g.xe[q * S + s] = st.xe[q];
      g.ve[q * S + s] = st.ve[q];
    }
    for (int q = t; q < N; q += L) {
      g.gsave[q * S + s] = gsv[tm][q];
      g.count[q * S + s] = cnt[tm][q];
    }
    if (t == 0 && !state_finite<N>(st)) atomicOr(g.status + s, NBG_STATUS_NONFINITE);
  }
}

// ------------------------------------------------------------ pairs on lanes
//
// Orbit producer for latency-bound chunks (up to lanes_limit systems of the
// group still running): one block per system (two systems of two or three
// bodies), sixteen lanes per pair solve.
// A warp issues one FP64 instruction per 64 cycles however independent its
// instructions are, and with few systems nothing else fills the SM, so a step
// takes as long as its longest warp's FP64 instructions; spreading a solve's
// independent pieces over lanes makes them one instruction each:
//   * lanes 0-5 hold the pair's relative coordinates, lanes 0-5 and 6-11 the
//     two bodies' (one subtraction, one Kahan sum instead of six and twelve);
//   * the three dot products, the two Stumpff polynomials, G2 and G3, G0 and
//     G1, Kepler's equation and r, and the four coefficients of the result are
//     evaluated side by side, each by its own lanes, and shuffled to all;
//   * the pairs of a level (equal i + j, see above) go to the block's half
//     warps, and phisalpha!'s pair terms to one lane each before each body sums
//     its own in pair order.
// 57 FP64 instructions a level instead of a one-lane solve's 146.  Every value is
// formed by the operations of kep_solve, phisalpha and kahan_fma in the same
// order, so the results are bitwise those of the other forms.
// One system alone, before (a pair solve on one lane or two) and after: 301 steps
// of five bodies without derivatives 30.2 -> 15.4 ms, 2000 steps of three bodies
// with transits 97 -> 67 ms (then bound by the consumer, jacobian_rows_kernel).
__host__ __device__ constexpr int lanes_warps(int N) { return (N / 2 + 1) / 2 > 0 ? (N / 2 + 1) / 2 : 1; }
// A level of two or three bodies has one pair: a system then takes a half warp.
__host__ __device__ constexpr int lanes_systems(int N) { return N <= 3 ? 2 : 1; }
__host__ __device__ constexpr int lanes_each(int N) { return 32 * lanes_warps(N) / lanes_systems(N); }

template <int N>
struct LanesShared {
  Sys<N> st;
  double a[3 * N], ac[3 * N], g[N];
  long long cnt[N];
  double pk[N * (N - 1) / 2], pmi[N * (N - 1) / 2], pmj[N * (N - 1) / 2];  // k, m_i / (m_i + m_j), m_j / (m_i + m_j)
  double f[N * (N - 1) / 2][3];
};

template <int N>
__device__ __forceinline__ void lanes_sync() {
  if (lanes_warps(N) == 1) __syncwarp();
  else __syncthreads();
}

// One pair of a sweep on the sixteen lanes hl = 0..15 of a half warp.  Both
// halves of a warp run the same instructions, so that its two pairs share their
// issue slots; a half without a pair (act false) repeats pair (0, 1) and writes
// nothing.  Only a solve that needs more than one FP64 step leaves the other
// half.
template <int N, bool DRIFT_FIRST>
__device__ __forceinline__ void lanes_pair(LanesShared<N>& sh, int i, int j, bool act, double h, const Rec& cap,
                                           int coff, int hl) {
  const int pb = pair_bit(i, j, N);
  const double k = sh.pk[pb];
  if (k == 0.0) {
    if (act && cap.p && hl == 0) cap.put(coff + PCAP_RINV, 0.0);
    act = false;
  }
  unsigned mask = 0xffffffffu;
  auto from = [&](double v, int src) { return __shfl_sync(mask, v, src, 16); };
  double* q = sh.st.x;  // x, v, xe, ve of Sys<N> in a row, 3N each
  const int c = hl % 6, k3 = hl % 3;
  const int at = (c < 3 ? 0 : 3 * N) + k3;
  const double qi = q[at + 3 * i], qj = q[at + 3 * j], d = qi - qj;
  // lanes 0-5 carry body i's coordinates, 6-11 body j's
  const int id = at + 3 * (hl < 6 ? i : j);
  double own_q = hl < 6 ? qi : qj, own_e = q[6 * N + id];
  const double weight = hl < 6 ? sh.pmj[pb] : -sh.pmi[pb];
  double X[3], V[3], R[3];
#pragma unroll
  for (int w = 0; w < 3; w++) {
    X[w] = from(d, w);
    V[w] = from(d, 3 + w);
  }
  const double xk = k3 == 0 ? X[0] : k3 == 1 ? X[1] : X[2], vk = k3 == 0 ? V[0] : k3 == 1 ? V[1] : V[2];
  if (DRIFT_FIRST) {
    const double rt = fma(-h, vk, xk);
#pragma unroll
    for (int w = 0; w < 3; w++) R[w] = from(rt, w);
  } else {
#pragma unroll
    for (int w = 0; w < 3; w++) R[w] = X[w];
  }
  double rr, vv, eta;
  {  // lanes by hl % 3: R.R, V.V, R.V
    double A[3], B[3];
#pragma unroll
    for (int w = 0; w < 3; w++) {
      A[w] = k3 == 1 ? V[w] : R[w];
      B[w] = k3 == 0 ? R[w] : V[w];
    }
    const double dot = fma(A[2], B[2], fma(A[1], B[1], A[0] * B[0]));
    rr = from(dot, 0);
    vv = from(dot, 1);
    eta = from(dot, 2);
  }
  const double r0inv = rsqrt_fast(rr);
  const double r0 = rr * r0inv;
  const double kr0 = k * r0inv;
  const double beta = fma(2.0, kr0, -vv);
  const double zeta = fma(-r0, beta, k);
  const double t = h * r0inv;
  float q2;
  const float sg = kep_start(to_float(r0inv), to_float(h), to_float(beta), to_float(eta), to_float(zeta), &q2);
  const double q2d = to_double(q2);
  const int w4 = hl & 3;
  const bool odd = hl & 1;
  double s = t * to_double(sg), ds, y, g0, g1, g2, g3, g4 = 0.0;
  bool done = false, far = false;
  auto iterate = [&]() {
    const double ss = s * s, z = beta * ss;
    const double scale = ss * (w4 == 0 ? 1.0 : w4 == 1 ? s : ss);
    const double g = scale * stumpff234(z, w4);  // G2, G3, G4 by w4
    g2 = from(g, 0);
    g3 = from(g, 1);
    if (!DRIFT_FIRST) g4 = from(g, 2);
    const double g01 = fma(-beta, odd ? g3 : g2, odd ? s : 1.0);
    g0 = from(g01, 0);
    g1 = from(g01, 1);
    const double first = fma(r0, s, -h);  // in the shuffles' shadow
    const double fr = fma(zeta, odd ? g2 : g3, fma(eta, odd ? g1 : g2, odd ? r0 : first));
    const double r = from(fr, 1);
    y = rcp_seed(r);
    const double ue = fma(odd ? -r : fr, y, odd ? 1.0 : 0.0);  // F / r to the seed's digits, and what they lack
    const double u = from(ue, 0);
    ds = -fma(u, fma(q2d, u, from(ue, 1)), u);
    s = s + ds;
    far = !(fabs(z) <= 4.0 * KEP_ZMAX);
    done = fabs(u) <= KEP_STEP * fabs(s) && fabs(z) <= KEP_ZMAX;
  };
  iterate();
  if (act && !done) {
    mask = 0xffffu << (threadIdx.x & 16);
    for (int iter = 1; iter < 6 && !done && !far; iter++) iterate();
    mask = 0xffffffffu;
  }
  __syncwarp();
  double del, val;  // val: fm1, gmh, dfdt, dgdtm1 by hl & 3
  KepParams P;
  {
    const double hd = 0.5 * ds;
    if (!DRIFT_FIRST) g4 = fma(ds, fma(hd, g2, g3), g4);
    const double gn = fma(ds, fma(hd, odd ? g1 : g0, odd ? g2 : g1), odd ? g3 : g2);
    g2 = from(gn, 0);
    g3 = from(gn, 1);
    g1 = fma(-beta, g3, s);
    const double r = fma(zeta, g2, fma(eta, g1, r0));
    const double rinv = rcp_from(r, y);
    const double krr = kr0 * rinv;
    double pre, mul;
    bool neg;
    if (DRIFT_FIRST) {
      const double ga = (w4 & 2) ? g1 : g2, gb = (w4 & 2) ? g2 : g3;
      const double both = fma(h, ga, -(r0 * gb));
      pre = (w4 & 2) ? krr : kr0;
      mul = (w4 & 1) ? both : ga;
      neg = !(w4 & 1);
    } else {
      const double kr = k * rinv;
      const double h12 = fma(s, odd ? g2 : g3, odd ? -g3 : -2.0 * g4);
      const double h1 = from(h12, 0), h2 = from(h12, 1);
      const double eh = eta * h1;
      const double ab = fma(w4 == 0 ? -kr0 : r0, w4 == 0 ? h1 : h2, w4 == 0 ? g2 : eh);
      pre = (w4 == 2) ? krr : kr;
      mul = (w4 < 2) ? ab : (w4 == 2) ? g1 : g2;
      neg = w4 >= 2;
    }
    val = pre * mul;
    if (neg) val = -val;
    P.s = s; P.g1 = g1; P.g2 = g2; P.g3 = g3; P.r0 = r0; P.r0inv = r0inv; P.rinv = rinv; P.beta = beta; P.eta = eta;
    P.zeta = zeta;
    const double cx = from(val, c < 3 ? 0 : 2), cv = from(val, c < 3 ? 1 : 3);
    del = fma(cx, xk, cv * vk);
  }
  if (act && !done) {
    double delxv[6];
    kep_solve_general<DRIFT_FIRST>(X, V, k, h, delxv, P);
    val = w4 == 0 ? P.fm1 : w4 == 1 ? P.gmh : w4 == 2 ? P.dfdt : P.dgdtm1;
    del = delxv[0];
#pragma unroll
    for (int w = 1; w < 6; w++) del = (c == w) ? delxv[w] : del;
  }
  if (act && hl < 12) {
    kahan_fma(own_q, own_e, weight, del);
    q[id] = own_q;
    q[6 * N + id] = own_e;
  }
  if (act && cap.p) {  // in put_capture's order: lanes 0-5 x0 and v0, 6-13 the solve, then 0-3 the coefficients
    double own = d;
    own = hl == 6 ? P.s : own;
    own = hl == 7 ? P.g2 : own;
    own = hl == 8 ? P.g3 : own;
    own = hl == 9 ? P.r0 : own;
    own = hl == 10 ? P.r0inv : own;
    own = hl == 11 ? P.rinv : own;
    own = hl == 12 ? P.beta : own;
    own = hl == 13 ? P.eta : own;
    double* to = cap.p + (unsigned)((coff + hl) * cap.stride);  // below 2^31: 2 P PCAP slots
    if (hl < 14) *to = own;
    if (hl < 4) to[(unsigned)(14 * cap.stride)] = val;
  }
}

// One AHL21 step on a system's lanes t (plain_step's values); run is false for
// the lanes of a system that does not step: they keep step with their warp and
// write nothing.  KICK: the group has kick pairs (kick).
template <int N, bool KICK>
__device__ __forceinline__ void lanes_step(LanesShared<N>& sh, int t, bool run, double h, uint64_t kick,
                                           const Rec& cap, const Rec& xs, const Rec& vs) {
  constexpr int P = N * (N - 1) / 2, T = lanes_each(N);
  static_assert(P <= T && 3 * N <= T, "one lane per pair and per coordinate");
  const int half = t >> 4, hl = t & 15;
  const double h2 = 0.5 * h;
  const bool coord = run && t < 3 * N, pair = run && t < P;
  Sys<N>& st = sh.st;
  int pi = 0, pj = t + 1;  // pair t's bodies
  while (pj >= N && pi < N - 2) {
    pi++;
    pj += pi + 1 - N;
  }
  const int b = t / 3, w = t % 3;  // coordinate lane
  const bool kicked = KICK && pair && ((kick >> t) & 1);
  auto pair_at = [&](int o) { return o < b ? pair_bit(o, b, N) : pair_bit(b, o, N); };
  auto is_kick = [&](int o) { return KICK && ((kick >> pair_at(o)) & 1); };
  double rij[3], r2 = 0.0, rinv = 0.0;
  auto force = [&](bool which) {  // G r / r^3 of pair t
    if (!which) return;
#pragma unroll
    for (int q = 0; q < 3; q++) rij[q] = st.x[3 * pi + q] - st.x[3 * pj + q];
    r2 = norm2(rij);
    rinv = rsqrt_fast(r2);
    phis_accel(rij, rinv, sh.f[t]);
  };
  auto kick_v = [&](double hk) {  // the kicked pairs' velocity changes, by body and in pair order
    if (!coord) return;
    double v = st.v[t], ve = st.ve[t];
    for (int o = 0; o < N; o++)
      if (o != b && is_kick(o)) kahan_fma(v, ve, o < b ? hk * st.m[o] : -(hk * st.m[o]), sh.f[pair_at(o)][w]);
    st.v[t] = v;
    st.ve[t] = ve;
  };
  if (KICK) {
    if (xs.p && coord) xs.put(3 * N + t, st.x[t]);
    force(kicked);
    lanes_sync<N>();
    kick_v(h / 6.0);
  }
  if (coord) {
    if (vs.p) vs.put(t, st.v[t]);
    kahan_fma(st.x[t], st.xe[t], h2, st.v[t]);
  }
  lanes_sync<N>();
  // a Kepler pair's capture slot: the ones before it in sweep order
  auto slot_of = [&](int pb) { return KICK ? pb - __popcll(kick & ((1ull << pb) - 1)) : pb; };
  const int npk = KICK ? P - __popcll(kick) : P;
#pragma unroll 1
  for (int lev = 1; lev <= 2 * N - 3; lev++) {
    int i = 0, j = 1;
    bool act = level_pair<N>(lev, half, &i, &j) && run;
    const int pb = pair_bit(i, j, N);
    if (KICK) act = act && !((kick >> pb) & 1);
    if (__any_sync(0xffffffffu, act)) lanes_pair<N, true>(sh, i, j, act, h2, cap, slot_of(pb) * PCAP, hl);
    lanes_sync<N>();
  }
  if (xs.p && coord) xs.put(t, st.x[t]);
  force(pair);
  lanes_sync<N>();
  if (KICK) kick_v(2.0 * h / 3.0);
  if (coord) {
    double a = 0.0, ac = 0.0;  // by the Kepler pairs and by the kicked ones
    for (int o = 0; o < N; o++)
      if (o != b) {
        const double f = sh.f[pair_at(o)][w], m = o < b ? st.m[o] : -st.m[o];
        if (is_kick(o)) ac = fma(m, f, ac);
        else a = fma(m, f, a);
      }
    sh.a[t] = a;
    if (KICK) sh.ac[t] = ac;
    if (xs.p && !KICK) xs.put(3 * N + t, a);
  }
  lanes_sync<N>();
  if (pair) {
    const double* a = kicked ? sh.ac : sh.a;
    double aij[3];
#pragma unroll
    for (int q = 0; q < 3; q++) aij[q] = a[3 * pi + q] - a[3 * pj + q];
    phis_corr(rij, r2, rinv, aij, kicked ? 0.0 : st.m[pi] + st.m[pj], kicked ? phic_coeff(h) : phis_coeff(h), sh.f[t]);
  }
  lanes_sync<N>();
  if (coord) {
    double v = st.v[t], ve = st.ve[t];
    for (int pass = KICK ? 0 : 1; pass < 2; pass++)  // the kicked pairs' corrections, then the Kepler pairs'
      for (int o = 0; o < N; o++)
        if (o != b && is_kick(o) == (pass == 0)) kahan_fma(v, ve, o < b ? -st.m[o] : st.m[o], sh.f[pair_at(o)][w]);
    st.v[t] = v;
    st.ve[t] = ve;
  }
  lanes_sync<N>();
#pragma unroll 1
  for (int lev = 2 * N - 3; lev >= 1; lev--) {
    int i = 0, j = 1;
    bool act = level_pair<N>(lev, half, &i, &j) && run;
    const int pb = pair_bit(i, j, N);
    if (KICK) act = act && !((kick >> pb) & 1);
    if (__any_sync(0xffffffffu, act))
      lanes_pair<N, false>(sh, i, j, act, h2, cap, (npk + (npk - 1 - slot_of(pb))) * PCAP, hl);
    lanes_sync<N>();
  }
  if (coord) {
    if (vs.p) vs.put(3 * N + t, st.v[t]);
    kahan_fma(st.x[t], st.xe[t], h2, st.v[t]);
  }
  lanes_sync<N>();
  if (KICK) {
    if (xs.p && coord) xs.put(6 * N + t, st.x[t]);
    force(kicked);
    lanes_sync<N>();
    kick_v(h / 6.0);
    lanes_sync<N>();
  }
}

template <int N, bool KICK>
__global__ void __launch_bounds__(32 * lanes_warps(N)) orbit_lanes_kernel(GroupArgs g, int chunk) {
  extern __shared__ double lanes_smem[];
  constexpr int P = N * (N - 1) / 2, T = lanes_each(N);
  const int t = threadIdx.x % T, S = g.S, s = blockIdx.x * lanes_systems(N) + threadIdx.x / T;
  LanesShared<N>& sh = reinterpret_cast<LanesShared<N>*>(lanes_smem)[threadIdx.x / T];
  bool valid = s < S && g.sysidx[s] >= 0;
  const long long nst = valid ? g.nsteps[s] : 0, k0 = valid ? chunk_first_step(g, chunk, s) : 0;
  valid = valid && k0 < nst && k0 >= 0;  // neither done nor admitted for a later chunk
  // the block's systems step together until the last of them has done
  const int nk = valid ? (int)(nst - k0 < g.K ? nst - k0 : g.K) : 0;
  const int most = lanes_systems(N) > 1 ? max(nk, __shfl_xor_sync(0xffffffffu, nk, 16)) : nk;
  if (most == 0) return;
  Sys<N>& st = sh.st;
  if (t < 3 * N) {
    st.x[t] = valid ? g.x[t * S + s] : 0.0;
    st.v[t] = valid ? g.v[t * S + s] : 0.0;
    st.xe[t] = valid ? g.xe[t * S + s] : 0.0;
    st.ve[t] = valid ? g.ve[t * S + s] : 0.0;
  }
  if (t < N) {
    st.m[t] = valid ? g.m[t * S + s] : 0.0;
    sh.g[t] = valid ? g.gsave[t * S + s] : 0.0;
    sh.cnt[t] = valid ? g.count[t * S + s] : 0;
  }
  lanes_sync<N>();
  if (t < P) {
    int i = 0, j = t + 1;
    while (j >= N && i < N - 2) {
      i++;
      j += i + 1 - N;
    }
    const double mij = st.m[i] + st.m[j], inv = rcp_fast(mij);
    sh.pk[t] = GNEWT * mij;
    sh.pmi[t] = st.m[i] * inv;
    sh.pmj[t] = st.m[j] * inv;
  }
  lanes_sync<N>();
  const double t0 = valid ? g.t0[s] : 0.0, h = valid ? g.h[s] : 0.0, hI = valid ? g.hI[s] : 0.0;
  const int ntt = valid ? g.ntt[s] : 0, ti = valid ? g.ti[s] : 0;
  for (int kk = 0; kk < most; kk++) {
    const long long istep = k0 + kk;
    const bool run = kk < nk;
    Rec cap{nullptr, 0}, xs{nullptr, 0};
    if (g.grad && run) {
      cap = Rec{g.pcap + (size_t)kk * 2 * g.npk * PCAP * S + s, S};
      xs = Rec{g.xsnap + (size_t)kk * snap_count(KICK) * 3 * N * S + s, S};
    }
    const double hs = run ? step_length(g, s, istep, nst, h) : h;
    if (g.trajxv && run && t < 3 * N) {
      double* rx = g.trajxv + ((size_t)s * g.K + kk) * 6 * N;
      rx[t] = st.x[t];
      rx[3 * N + t] = st.v[t];
    }
    const Rec vs{g.grad && run && istep == nst - 1 ? g.vsnap + s : nullptr, S};
    lanes_step<N, KICK>(sh, t, run, hs, g.kick, cap, xs, vs);
    if (!g.notransit && run && t < N - 1)
      detect_transit<N>(g, st, s, kk, t, ti, ntt, hI, t0 + (double)(istep + 1) * h, sh.g, sh.cnt);
    lanes_sync<N>();
  }
  if (!valid) return;
  if (t < 3 * N) {
    g.x[t * S + s] = st.x[t];
    g.v[t * S + s] = st.v[t];
    g.xe[t * S + s] = st.xe[t];
    g.ve[t * S + s] = st.ve[t];
  }
  if (t < N) {
    g.gsave[t * S + s] = sh.g[t];
    g.count[t * S + s] = sh.cnt[t];
  }
  if (t == 0 && !state_finite<N>(st)) atomicOr(g.status + s, NBG_STATUS_NONFINITE);
}

}  // namespace nbg
