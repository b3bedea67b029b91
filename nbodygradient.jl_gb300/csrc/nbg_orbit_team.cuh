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
      kahan(s.x[q], s.xe[q], h2 * s.v[q]);
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
      kahan(s.x[q], s.xe[q], h2 * s.v[q]);
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
// group still running): one block per system and one warp per pair of a level,
// or two systems of two or three bodies (whose levels have one pair) to a warp.
// A warp issues one FP64 instruction per 64 cycles however independent its
// instructions are, and with few systems nothing else fills the SM, so a step
// takes as long as its longest warp's FP64 instructions; spreading a solve's
// independent pieces over sixteen lanes makes them one instruction each:
//   * lanes 0-5 hold the pair's relative coordinates, lanes 0-5 and 6-11 the
//     two bodies' (one subtraction, one Kahan sum instead of six and twelve);
//   * the three dot products, 1 / beta and 6 / zeta, the cubic's coefficients,
//     the sine and cosine series, numerator and denominator of the Newton
//     update, G1, G3, H1 and H2, the sum of r and the four coefficients of the
//     result are evaluated side by side, each by its own lanes, and shuffled to
//     all;
//   * phisalpha!'s pair terms go to one lane each before each body sums its own
//     in pair order.
// Every value is formed by the operations of kep_solve, phisalpha and kahan in
// the same order, so the results are bitwise those of the other forms.  From
// four bodies on a pair has a warp, whose upper lanes repeat the lower ones and
// write nothing (an FP64 instruction costs the same): a bound and a hyperbolic
// pair in one warp would wait for each other.
// One system alone, a solve on one lane or two -> here: 301 steps of five bodies
// without derivatives 84 -> 56 ms, 400 of eight with transits 261 -> 146 ms.
__host__ __device__ constexpr int lanes_warps(int N) { return N <= 3 ? 1 : N / 2; }
// A level of two or three bodies has one pair: a system then takes a half warp.
__host__ __device__ constexpr int lanes_systems(int N) { return N <= 3 ? 2 : 1; }
__host__ __device__ constexpr int lanes_each(int N) { return 32 * lanes_warps(N) / lanes_systems(N); }

template <int N>
struct LanesShared {
  Sys<N> st;
  double a[3 * N], ac[3 * N], g[N];
  long long cnt[N];
  double pk[N * (N - 1) / 2], pmi[N * (N - 1) / 2], pmj[N * (N - 1) / 2];  // k, m_i / (m_i + m_j), m_j / (m_i + m_j)
  double f[N * (N - 1) / 2][3], fk[N * (N - 1) / 2][3];
};

template <int N>
__device__ __forceinline__ void lanes_sync() {
  if (lanes_warps(N) == 1) __syncwarp();
  else __syncthreads();
}

// The coefficients of G3, H1 and H2 (kGHCoef), by lane.
template <int Q>
__device__ __forceinline__ double gh_coef(int n) {
  constexpr double g3[11] = {0x1.0000000000000p+0, 0x1.999999999999ap-5, 0x1.3813813813814p-10, 0x1.1566abc011567p-16, 0x1.42cb40df7f3abp-23, 0x1.08db48ebe51c7p-30, 0x1.42df6ed66ca17p-38, 0x1.2fe15942481f8p-46, 0x1.c6ee8e9c1e203p-55, 0x1.154ab3925b815p-63, 0x1.189470e50aa13p-72};
  constexpr double h1[11] = {0x1.0000000000000p+0, 0x1.1111111111111p-4, 0x1.d41d41d41d41dp-10, 0x1.bbd779334ef0bp-16, 0x1.0cfeb60f94b0ep-22, 0x1.c60a33dd88c31p-30, 0x1.1a8380fb9f0d4p-37, 0x1.0e1da4acb1e32p-45, 0x1.99704d261b1cfp-54, 0x1.f82abadb8f19bp-63, 0x1.0132bcd1f4692p-71};
  constexpr double h2[11] = {0x1.0000000000000p+0, 0x1.999999999999ap-4, 0x1.d41d41d41d41dp-9, 0x1.1566abc011567p-14, 0x1.937e11175f095p-21, 0x1.8d48ed61d7aabp-28, 0x1.1a8380fb9f0d4p-35, 0x1.2fe15942481f8p-43, 0x1.ffcc606fa1e43p-52, 0x1.5a9d6076f261ap-60, 0x1.81cc1b3aee9dbp-69};
  return n == 0 ? g3[Q] : n == 1 ? h1[Q] : h2[Q];
}
template <int Q>
__device__ __forceinline__ double gh_horner_of(int n, double x2, double p) {
  p = fma(p, x2, gh_coef<Q>(n));
  if constexpr (Q > 0) return gh_horner_of<Q - 1>(n, x2, p);
  return p;
}

// One pair of a sweep on the sixteen lanes hl = 0..15 of a half warp.  The whole
// warp runs the same instructions: its other half has the other system's pair
// (N <= 3) or repeats this one (write false).  A half without a pair (act
// false) repeats pair (0, 1) of its own system and writes nothing.
template <int N, bool DRIFT_FIRST>
__device__ __forceinline__ void lanes_pair(LanesShared<N>& sh, int i, int j, bool act, double h, const Rec& cap,
                                           int coff, int hl, bool write) {
  constexpr unsigned ALL = 0xffffffffu;
  const int pb = pair_bit(i, j, N);
  const double k = sh.pk[pb];
  if (k == 0.0) {
    if (act && write && cap.p && hl == 0) cap.put(coff + PCAP_RINV, 0.0);
    act = false;
  }
  if (!__any_sync(ALL, act)) return;
  auto from = [](double v, int src) { return __shfl_sync(ALL, v, src, 16); };
  double* q = sh.st.x;  // x, v, xe, ve of Sys<N> in a row, 3N each
  const int c = hl % 6, k3 = hl % 3, w4 = hl & 3;
  const bool odd = hl & 1;
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
    const double rt = xk - h * vk;
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
    const double dot = A[0] * B[0] + A[1] * B[1] + A[2] * B[2];
    rr = from(dot, 0);
    vv = from(dot, 1);
    eta = from(dot, 2);
  }
  const double r0 = sqrt(rr);
  const double r0inv = 1.0 / r0;
  const double beta = 2.0 * k * r0inv - vv;
  const double signb = jsign(beta);
  const bool plus = signb > 0.0;  // products with signb = +-1 are changes of sign
  const double sqb = sqrt(signb * beta);
  const double rb = r0 * beta;
  const double zeta = k - rb;
  // the solve's other branches (zeta or beta zero): all of it on every lane
  const bool plain = act && !(zeta != 0.0 && beta != 0.0);
  const bool solve = act && !plain;
  double betainv, gamma;
  {
    const double inv = (odd ? 6.0 : 1.0) / (odd ? zeta : beta);
    betainv = from(inv, 0);
    const double zinv = from(inv, 1);
    const double hs = plus ? -h : h;
    // cubic1's arguments a, b, c on lanes 0, 1, 2
    const double first = (w4 == 2 ? hs : 0.5) * (w4 == 2 ? beta : eta);
    const double arg = ((w4 == 1 ? rb : first) * (w4 == 1 ? signb : sqb)) * zinv;
    const double third = arg * THIRD;
    const double b = from(arg, 1), cc = from(arg, 2), a3 = from(third, 0);
    const double a3sq = a3 * a3;
    const double Q = a3sq - from(third, 1);
    const double pr = (odd ? -a3 : a3sq) * (odd ? b : a3);
    const double Rc = from(pr, 0) + 0.5 * (from(pr, 1) + cc);
    const double sq = (odd ? Q : Rc) * (odd ? Q : Rc);
    const double R2 = from(sq, 0), Q3 = from(sq, 1) * Q;
    if (R2 < Q3) {
      gamma = -cc / b;
    } else {
      const double A = (-jsign(Rc)) * cbrt(fabs(Rc) + sqrt(R2 - Q3));
      const double B = (A == 0.0) ? 0.0 : Q / A;
      gamma = A + B - a3;
    }
  }
  // the Newton update's numerator on even lanes, its denominator on odd ones
  const double e2 = plus ? 2.0 * eta : -(2.0 * eta);
  const double pc = sqb * (odd ? h : e2);
  const double c3 = from(pc, 0), c4 = -from(pc, 1) * beta;
  const double z2 = 2.0 * zeta;
  const double a1 = odd ? (plus ? z2 : -z2) : k, a2 = odd ? c3 : -z2;
  const bool ell = beta > 0.0;
  const bool any_ell = __any_sync(ALL, solve && ell), any_hyp = __any_sync(ALL, solve && !ell);
  double sx = 0.0, cx = 0.0;
  auto functions = [&](double x) {  // sine and cosine of x, or their hyperbolic counterparts
    if (any_ell) {
      const double x2 = x * x;
      double p = odd ? -0x1.6827863b97d97p-53 : 0x1.952c77030ad4ap-49;
      p = fma(p, x2, odd ? 0x1.ae7f3e733b81fp-45 : -0x1.ae7f3e733b81fp-41);
      p = fma(p, x2, odd ? -0x1.93974a8c07c9dp-37 : 0x1.6124613a86d09p-33);
      p = fma(p, x2, odd ? 0x1.1eed8eff8d898p-29 : -0x1.ae64567f544e4p-26);
      p = fma(p, x2, odd ? -0x1.27e4fb7789f5cp-22 : 0x1.71de3a556c734p-19);
      p = fma(p, x2, odd ? 0x1.a01a01a01a01ap-16 : -0x1.a01a01a01a01ap-13);
      p = fma(p, x2, odd ? -0x1.6c16c16c16c17p-10 : 0x1.1111111111111p-7);
      p = fma(p, x2, odd ? 0x1.5555555555555p-5 : -0x1.5555555555555p-3);
      const double b = x2 * (odd ? x2 : x);
      const double one = fma(-0.5, x2, 1.0);
      const double v = fma(b, p, odd ? one : x);
      sx = from(v, 0);
      cx = from(v, 1);
      if (ell && fabs(x) > 0.78539816339744831) sincos(x, &sx, &cx);
    }
    if (any_hyp && !ell) {
      sx = sinh(x);
      cx = exp(-x) + sx;
    }
  };
  {
    double gamma1 = 2.0 * gamma, gamma2 = 3.0 * gamma;
    int iter = 0;
    bool done = !solve;
#pragma unroll 1
    while (__any_sync(ALL, !done)) {
      if (!done) {
        gamma2 = gamma1;
        gamma1 = gamma;
      }
      functions(0.5 * gamma);
      const double ss = sx * sx;
      double acc = a1 * (odd ? ss : gamma) + (a2 * sx) * cx;
      acc = acc + (odd ? rb : c3 * ss);
      const double acc4 = acc + c4;
      acc = odd ? acc : acc4;
      const double num = from(acc, 0), den = from(acc, 1);
      const double next = gamma - num / den;
      if (!done) {
        gamma = next;
        iter += 1;
        done = iter >= 20 || gamma == gamma2 || gamma == gamma1;
      }
    }
  }
  functions(0.5 * gamma);
  const bool big = solve && !(gamma < 0.5);
  double g0, g1, g2, g3, h1 = 0.0, h2 = 0.0;
  {  // lanes by w4: G3, H1, H2 and, on 3, G2, beta G2 and G1
    const double sq = (w4 == 3 ? sx : gamma) * (w4 == 3 ? sx : gamma);
    const double x2 = plus ? -sq : sq, s2 = plus ? 2.0 * sq : -(2.0 * sq);
    const double p1 = (w4 == 3 ? s2 : w4 == 1 ? beta : w4 == 0 ? 6.0 : 3.0) * (w4 == 3 ? betainv : beta);
    g2 = from(p1, 3);
    const double p2 = (w4 == 3 ? beta : p1) * (w4 == 3 ? g2 : w4 == 1 ? 12.0 : sqb);
    g0 = 1.0 - from(p2, 3);
    const double num = (w4 == 3 ? 2.0 * sx : w4 == 1 ? x2 : -x2) * (w4 == 3 ? cx : w4 == 1 ? x2 : gamma);
    const double quot = num / (w4 == 3 ? sqb : p2);
    g1 = from(quot, 3);
    const double val = gh_horner_of<9>(w4, x2, gh_coef<10>(w4)) * quot;
    g3 = from(val, 0);
    if (!DRIFT_FIRST) {
      h1 = from(val, 1);
      h2 = from(val, 2);
    }
    if (big) {
      const GH gh = gh_functions<DRIFT_FIRST ? GH_G3 : (GH_G3 | GH_H1 | GH_H2)>(gamma, beta, sqb);
      g3 = gh.g3;
      h1 = gh.h1;
      h2 = gh.h2;
    }
    __syncwarp();
  }
  const double rp = (w4 == 0 ? r0 : w4 == 1 ? eta : k) * (w4 == 0 ? g0 : w4 == 1 ? g1 : g2);
  const double r = from(rp, 0) + from(rp, 1) + from(rp, 2);
  const double rinv = 1.0 / r;
  double val;  // fm1, gmh, dfdt, dgdtm1 by w4
  if (DRIFT_FIRST) {
    double pre = ((w4 & 1) ? k : -k) * (w4 == 2 ? g1 : r0inv);
    const double pr = pre * rinv;
    pre = (w4 & 2) ? pr : pre;
    const double a = h * (w4 == 1 ? g2 : g1), b = r0 * (w4 == 1 ? g3 : g2);
    val = pre * (w4 == 0 ? g2 : w4 == 2 ? r0inv : a - b);
  } else {
    double pre = (w4 < 2 ? k : -k) * (w4 == 2 ? g1 : rinv);
    const double pr = pre * rinv;
    pre = w4 == 2 ? pr : pre;
    const double a = (w4 == 0 ? k : eta) * (w4 == 0 ? r0inv : h1);
    const double b = (w4 == 0 ? a : r0) * (w4 == 0 ? h1 : h2);
    const double in = (w4 == 0 ? g2 : a) + (w4 == 0 ? -b : b);
    val = pre * (w4 < 2 ? in : w4 == 2 ? r0inv : g2);
  }
  double del;
  {  // the products with x0 on lanes 0-5, with v0 on 6-11
    const double prod = from(val, (c < 3 ? 0 : 2) + (hl < 6 ? 0 : 1)) * (hl < 6 ? xk : vk);
    del = from(prod, c) + from(prod, 6 + c);
  }
  double cg = gamma, cg2 = g2, cg3 = g3, crinv = rinv;
  if (plain) {
    KepParams P;
    double delxv[6];
    kep_solve<DRIFT_FIRST>(X, V, k, h, delxv, P);
    val = w4 == 0 ? P.fm1 : w4 == 1 ? P.gmh : w4 == 2 ? P.dfdt : P.dgdtm1;
    cg = P.gamma;
    cg2 = P.g2;
    cg3 = P.g3;
    crinv = P.rinv;
    del = delxv[0];
#pragma unroll
    for (int w = 1; w < 6; w++) del = (c == w) ? delxv[w] : del;
  }
  if (act && write && hl < 12) {
    kahan(own_q, own_e, weight * del);
    q[id] = own_q;
    q[6 * N + id] = own_e;
  }
  if (act && write && cap.p) {  // in put_capture's order: lanes 0-5 x0 and v0, 6-13 the solve, then 0-3 the coefficients
    double own = d;
    own = hl == 6 ? cg : own;
    own = hl == 7 ? cg2 : own;
    own = hl == 8 ? cg3 : own;
    own = hl == 9 ? r0 : own;
    own = hl == 10 ? r0inv : own;
    own = hl == 11 ? crinv : own;
    own = hl == 12 ? beta : own;
    own = hl == 13 ? eta : own;
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
  const int slot = t / (N <= 3 ? 16 : 32), hl = t & 15;
  const bool write = N <= 3 || !(t & 16);
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
  double rij[3], r2 = 0.0, r1 = 0.0;
  auto apart = [&]() {
#pragma unroll
    for (int q = 0; q < 3; q++) rij[q] = st.x[3 * pi + q] - st.x[3 * pj + q];
  };
  auto kick_force = [&](double hk) {  // of pair t over hk
    if (!kicked) return;
    apart();
    const double fac2 = hk * GNEWT * kick_r3inv(rij);
#pragma unroll
    for (int q = 0; q < 3; q++) sh.fk[t][q] = fac2 * rij[q];
  };
  auto kick_v = [&]() {  // the kicked pairs' velocity changes, by body and in pair order
    if (!coord) return;
    double v = st.v[t], ve = st.ve[t];
    for (int o = 0; o < N; o++)
      if (o != b && is_kick(o)) kahan(v, ve, (o < b ? st.m[o] : -st.m[o]) * sh.fk[pair_at(o)][w]);
    st.v[t] = v;
    st.ve[t] = ve;
  };
  if (KICK) {
    if (xs.p && coord) xs.put(3 * N + t, st.x[t]);
    kick_force(h / 6.0);
    lanes_sync<N>();
    kick_v();
  }
  if (coord) {
    if (vs.p) vs.put(t, st.v[t]);
    kahan(st.x[t], st.xe[t], h2 * st.v[t]);
  }
  lanes_sync<N>();
  // a Kepler pair's capture slot: the ones before it in sweep order
  auto slot_of = [&](int pb) { return KICK ? pb - __popcll(kick & ((1ull << pb) - 1)) : pb; };
  const int npk = KICK ? P - __popcll(kick) : P;
#pragma unroll 1
  for (int lev = 1; lev <= 2 * N - 3; lev++) {
    int i = 0, j = 1;
    bool act = level_pair<N>(lev, slot, &i, &j) && run;
    const int pb = pair_bit(i, j, N);
    if (KICK) act = act && !((kick >> pb) & 1);
    if (__any_sync(0xffffffffu, act)) lanes_pair<N, true>(sh, i, j, act, h2, cap, slot_of(pb) * PCAP, hl, write);
    lanes_sync<N>();
  }
  if (xs.p && coord) xs.put(t, st.x[t]);
  if (pair) {
    apart();
    r2 = norm2(rij);
    r1 = sqrt(r2);
    if (kicked) {
      const double r3inv = kick_r3inv(rij);
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const double fac = GNEWT * rij[q] * r3inv;
        sh.f[t][q] = fac;
        sh.fk[t][q] = fac * 2.0 * h / 3.0;
      }
    } else {
      phis_accel(rij, r2, r1, sh.f[t]);
    }
  }
  lanes_sync<N>();
  if (KICK) kick_v();
  if (coord) {
    double a = 0.0, ac = 0.0;  // by the Kepler pairs and by the kicked ones
    for (int o = 0; o < N; o++)
      if (o != b) {
        const double f = sh.f[pair_at(o)][w], m = o < b ? st.m[o] : -st.m[o];
        if (is_kick(o)) ac = ac + m * f;
        else a = a + m * f;
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
    phis_corr(rij, r2, r1, aij, kicked ? 0.0 : st.m[pi] + st.m[pj], kicked ? phic_coeff(h) : phis_coeff(h), sh.f[t]);
  }
  lanes_sync<N>();
  if (coord) {
    double v = st.v[t], ve = st.ve[t];
    for (int pass = KICK ? 0 : 1; pass < 2; pass++)  // the kicked pairs' corrections, then the Kepler pairs'
      for (int o = 0; o < N; o++)
        if (o != b && is_kick(o) == (pass == 0)) kahan(v, ve, (o < b ? -st.m[o] : st.m[o]) * sh.f[pair_at(o)][w]);
    st.v[t] = v;
    st.ve[t] = ve;
  }
  lanes_sync<N>();
#pragma unroll 1
  for (int lev = 2 * N - 3; lev >= 1; lev--) {
    int i = 0, j = 1;
    bool act = level_pair<N>(lev, slot, &i, &j) && run;
    const int pb = pair_bit(i, j, N);
    if (KICK) act = act && !((kick >> pb) & 1);
    if (__any_sync(0xffffffffu, act))
      lanes_pair<N, false>(sh, i, j, act, h2, cap, (npk + (npk - 1 - slot_of(pb))) * PCAP, hl, write);
    lanes_sync<N>();
  }
  if (coord) {
    if (vs.p) vs.put(3 * N + t, st.v[t]);
    kahan(st.x[t], st.xe[t], h2 * st.v[t]);
  }
  lanes_sync<N>();
  if (KICK) {
    if (xs.p && coord) xs.put(6 * N + t, st.x[t]);
    kick_force(h / 6.0);
    lanes_sync<N>();
    kick_v();
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
  // a slot without a system beside one that runs gets ordinary numbers: division
  // and square root of a zero or a NaN leave the short path, and its half warp
  // runs with the other's
  if (t < 3 * N) {
    st.x[t] = valid ? g.x[t * S + s] : (t % 3 == 0) ? t / 3 : 0.0;
    st.v[t] = valid ? g.v[t * S + s] : (t % 3 == 1) ? 0.01 * (t / 3) : 0.0;
    st.xe[t] = valid ? g.xe[t * S + s] : 0.0;
    st.ve[t] = valid ? g.ve[t * S + s] : 0.0;
  }
  if (t < N) {
    st.m[t] = valid ? g.m[t * S + s] : 1.0;
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
    const double mij = st.m[i] + st.m[j], inv = 1.0 / mij;
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
