// nbg_kepler.cuh -- device-side universal-variable Kepler drift for one body
// pair and its analytic Jacobian, FP64.
//
// Restates, for one lane = one system, NbodyGradient.jl's
//   jac_delxv_gamma!        src/integrator/ahl21/ahl21.jl:766-890
//   compute_jacobian_gamma! src/integrator/ahl21/ahl21.jl:896-1139
//   cubic1, G3, H1, H2 and their series  src/utils.jl:103-396
// The translation unit is compiled with --fmad=false: every product and sum
// rounds on its own but where fma() is written.
//
// What moves x and v (kep_solve, and the steps in nbg_orbit.cuh) rounds
// operation by operation as the reference's expressions do, with correctly
// rounded division and square root: whether a transit search's iterates repeat
// within their limit hangs on the last digit of x and v, and with it the
// status word NBG_STATUS_NEWTON_ITMAX.  What only the Jacobian reads
// (kep_derivatives and on) is free in its rounding and takes fused products and
// reciprocals of one ulp.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nbg {

// src/NbodyGradient.jl:13-17
constexpr double GNEWT = 39.4845 / (365.242 * 365.242);
constexpr double THIRD = 1.0 / 3.0;

__device__ __forceinline__ double jsign(double x) { return x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : x); }

// comp_sum (src/utils.jl:16-23)
__device__ __forceinline__ void kahan(double& s, double& e, double a) {
  e = e + a;
  double t = s + e;
  e = (s - t) + e;
  s = t;
}

// 1/x and 1/sqrt(x) to about one ulp from the hardware's seeds (PTX
// rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64) by one step of Householder's
// cubically convergent iteration on e = 1 - x y and e = 1 - x y^2: three and
// five FP64 instructions.  A zero gives NaN, not infinity: callers divide by
// what is zero in no valid state.
__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// one step from an estimate y of 1/x
__device__ __forceinline__ double rcp_from(double x, double y) {
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rcp_fast(double x) { return rcp_from(x, rcp_seed(x)); }
__device__ __forceinline__ double rsqrt_fast(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// cubic1 (src/utils.jl:103-122)
__device__ __forceinline__ double cubic1(double a, double b, double c) {
  double a3 = a * THIRD;
  double Q = a3 * a3 - b * THIRD;
  double R = a3 * a3 * a3 + 0.5 * ((-a3) * b + c);
  double R2 = R * R, Q3 = Q * Q * Q;
  if (R2 < Q3) return -c / b;
  double A = (-jsign(R)) * cbrt(fabs(R) + sqrt(R2 - Q3));
  double B = (A == 0.0) ? 0.0 : Q / A;
  return A + B - a3;
}

// sin and cos of |x| <= pi/4 from their Taylor series about 0 (coefficients
// (-1)^k / (2k+1)! up to x^17 and (-1)^k / (2k)! up to x^18, Horner scheme in
// x^2).  The truncation error at |x| = pi/4 is below 1e-19, the evaluation
// error about one ulp; the result is checked against CUDA's sin and cos
// (tests/test_gpu_math.py).  Outside |x| <= pi/4 CUDA's sincos is used.
// The half-angle x = gamma / 2 of the Kepler solve is far below pi/4 for
// bound orbits stepped at a fraction of their period.
__device__ __forceinline__ void sincos_kepler(double x, double* s, double* c) {
  if (fabs(x) > 0.78539816339744831) {
    sincos(x, s, c);
    return;
  }
  const double x2 = x * x;
  double ps = 0x1.952c77030ad4ap-49;
  ps = fma(ps, x2, -0x1.ae7f3e733b81fp-41);
  ps = fma(ps, x2, 0x1.6124613a86d09p-33);
  ps = fma(ps, x2, -0x1.ae64567f544e4p-26);
  ps = fma(ps, x2, 0x1.71de3a556c734p-19);
  ps = fma(ps, x2, -0x1.a01a01a01a01ap-13);
  ps = fma(ps, x2, 0x1.1111111111111p-7);
  ps = fma(ps, x2, -0x1.5555555555555p-3);
  *s = fma(x * x2, ps, x);
  double pc = -0x1.6827863b97d97p-53;
  pc = fma(pc, x2, 0x1.ae7f3e733b81fp-45);
  pc = fma(pc, x2, -0x1.93974a8c07c9dp-37);
  pc = fma(pc, x2, 0x1.1eed8eff8d898p-29);
  pc = fma(pc, x2, -0x1.27e4fb7789f5cp-22);
  pc = fma(pc, x2, 0x1.a01a01a01a01ap-16);
  pc = fma(pc, x2, -0x1.6c16c16c16c17p-10);
  pc = fma(pc, x2, 0x1.5555555555555p-5);
  *c = fma(x2 * x2, pc, fma(-0.5, x2, 1.0));
}

enum : int { GH_G3 = 1, GH_H1 = 2, GH_H2 = 4 };

struct GH {
  double g3, h1, h2;
};

// Coefficients c_n of the G3, H1, H2, H3, H5, H6 series in x2 = -sign(beta) gamma^2
// (src/utils.jl:137-396), exact rationals rounded to double, n = 0..10.
__device__ __constant__ double kGHCoef[6][11] = {
    {0x1.0000000000000p+0, 0x1.999999999999ap-5, 0x1.3813813813814p-10, 0x1.1566abc011567p-16, 0x1.42cb40df7f3abp-23, 0x1.08db48ebe51c7p-30, 0x1.42df6ed66ca17p-38, 0x1.2fe15942481f8p-46, 0x1.c6ee8e9c1e203p-55, 0x1.154ab3925b815p-63, 0x1.189470e50aa13p-72},  // G3
    {0x1.0000000000000p+0, 0x1.1111111111111p-4, 0x1.d41d41d41d41dp-10, 0x1.bbd779334ef0bp-16, 0x1.0cfeb60f94b0ep-22, 0x1.c60a33dd88c31p-30, 0x1.1a8380fb9f0d4p-37, 0x1.0e1da4acb1e32p-45, 0x1.99704d261b1cfp-54, 0x1.f82abadb8f19bp-63, 0x1.0132bcd1f4692p-71},  // H1
    {0x1.0000000000000p+0, 0x1.999999999999ap-4, 0x1.d41d41d41d41dp-9, 0x1.1566abc011567p-14, 0x1.937e11175f095p-21, 0x1.8d48ed61d7aabp-28, 0x1.1a8380fb9f0d4p-35, 0x1.2fe15942481f8p-43, 0x1.ffcc606fa1e43p-52, 0x1.5a9d6076f261ap-60, 0x1.81cc1b3aee9dbp-69},  // H2
    {0x1.999999999999ap-4, 0x1.8618618618618p-7, 0x1.6c16c16c16c17p-11, 0x1.acb5f228d4f9fp-16, 0x1.60cc1822382eep-21, 0x1.ae64567f544e4p-27, 0x1.952622512ec88p-33, 0x1.2f48851e5fad6p-39, 0x1.71b892ff937bap-46, 0x1.761b29cfaf6e8p-53, 0x1.3f3cc8d472c34p-60},  // H3
    {0x1.1111111111111p-6, 0x1.a01a01a01a01ap-11, 0x1.1566abc011567p-16, 0x1.ae64567f544e4p-23, 0x1.b96d79892884cp-30, 0x1.42df6ed66ca17p-37, 0x1.6286e822a97a1p-45, 0x1.2f49b46814157p-53, 0x1.9ff00d5b89420p-62, 0x1.d3a2117dbc620p-71, 0x1.b6f39affec388p-80},  // H5
    {0x1.999999999999ap-6, 0x1.5f15f15f15f16p-9, 0x1.18de5ab277f45p-13, 0x1.1a71d8c38f535p-18, 0x1.91b806e381809p-24, 0x1.adeb42b5c3e58p-30, 0x1.68045a5f7c07ap-36, 0x1.e535756d08617p-43, 0x1.0ce18de28b3bep-49, 0x1.f2cdf899367f3p-57, 0x1.88e826fd0f0dep-64},  // H6
};

__device__ __forceinline__ double gh_horner(const double* c, double x2) {
  double p = c[10];
#pragma unroll
  for (int n = 9; n >= 0; n--) p = fma(p, x2, c[n]);
  return p;
}

// G3, H1, H2 at (gamma, beta) -- the subset named by NEED.
// gamma < 0.5: the series of utils.jl:137-396 in x2 = -sign(beta) gamma^2,
// |x2| < 0.25, evaluated as degree-10 polynomials with the exact series
// coefficients (terms beyond n = 10 are below 1e-17 of the leading term).
// The reference sums term by term until the partial sum stops changing;
// the polynomial reaches the same value to rounding, without the series'
// dependent FP64 divisions.  gamma >= 0.5: the closed forms of utils.jl.
template <int NEED>
__device__ __forceinline__ GH gh_functions(double gamma, double beta, double sqb) {
  GH o;
  o.g3 = o.h1 = o.h2 = 0.0;
  if (gamma < 0.5) {
    const double x2 = (-jsign(beta)) * (gamma * gamma);
    if (NEED & GH_G3) o.g3 = gh_horner(kGHCoef[0], x2) * (((-x2) * gamma) / ((6.0 * beta) * sqb));
    if (NEED & GH_H1) o.h1 = gh_horner(kGHCoef[1], x2) * ((x2 * x2) / (12.0 * (beta * beta)));
    if (NEED & GH_H2) o.h2 = gh_horner(kGHCoef[2], x2) * (((-x2) * gamma) / ((3.0 * beta) * sqb));
  } else if (beta >= 0.0) {
    double s, c;
    sincos(gamma, &s, &c);
    if (NEED & GH_G3) o.g3 = (gamma - s) / (sqb * beta);
    if (NEED & GH_H1) {
      double sh = sin(0.5 * gamma);
      o.h1 = (4.0 * (sh * sh) - gamma * s) / (beta * beta);
    }
    if (NEED & GH_H2) o.h2 = (s - gamma * c) / (sqb * beta);
  } else {
    double s = sinh(gamma), c = cosh(gamma);
    if (NEED & GH_G3) o.g3 = (gamma - s) / (sqb * beta);
    if (NEED & GH_H1) {
      double sh = sinh(0.5 * gamma);
      o.h1 = (-4.0 * (sh * sh) + gamma * s) / (beta * beta);
    }
    if (NEED & GH_H2) o.h2 = (s - gamma * c) / (sqb * beta);
  }
  return o;
}

// What a drift leaves for its Jacobian (jac_delxv_gamma! returns the same
// quantities, ahl21.jl:888): gamma = s sqrt|beta| and the functions of it.
struct KepParams {
  double gamma, g1, g2, g3, dfdt, fm1, gmh, dgdtm1, r0, r, r0inv, rinv, k, h, beta, eta, zeta;
};

// jac_delxv_gamma! (ahl21.jl:766-890): Kepler drift of the relative orbit
// (x0, v0) with k = G (m_i + m_j) over h; writes delxv (position and velocity
// differences, finish - start minus the drift terms).
template <bool DRIFT_FIRST>
__device__ __noinline__ void kep_solve(const double* x0, const double* v0, double k, double h, double* delxv,
                                       KepParams& P) {
  double rt0 = x0[0] - h * v0[0], rt1 = x0[1] - h * v0[1], rt2 = x0[2] - h * v0[2];
  double r0 = DRIFT_FIRST ? sqrt(rt0 * rt0 + rt1 * rt1 + rt2 * rt2) : sqrt(x0[0] * x0[0] + x0[1] * x0[1] + x0[2] * x0[2]);
  double r0inv = 1.0 / r0;
  double beta0 = 2.0 * k * r0inv - (v0[0] * v0[0] + v0[1] * v0[1] + v0[2] * v0[2]);
  double beta0inv = 1.0 / beta0;
  double signb = jsign(beta0);
  double sqb = sqrt(signb * beta0);
  double zeta = k - r0 * beta0;
  double eta = DRIFT_FIRST ? (rt0 * v0[0] + rt1 * v0[1] + rt2 * v0[2]) : (x0[0] * v0[0] + x0[1] * v0[1] + x0[2] * v0[2]);
  double gamma_guess;
  if (zeta != 0.0) {
    double zinv = 6.0 / zeta;
    gamma_guess = cubic1(0.5 * eta * sqb * zinv, r0 * signb * beta0 * zinv, (-h) * signb * beta0 * sqb * zinv);
  } else if (eta != 0.0) {
    double reta = r0 / eta;
    double disc = reta * reta + 2.0 * h / eta;
    gamma_guess = (disc > 0.0) ? sqb * ((-reta) + sqrt(disc)) : h * r0inv * sqb;
  } else {
    gamma_guess = h * r0inv * sqb;
  }
  double gamma = gamma_guess;
  double gamma1 = 2.0 * gamma, gamma2 = 3.0 * gamma;
  double c2 = -2.0 * zeta, c3 = 2.0 * eta * signb * sqb, c4 = (-sqb) * h * beta0, c5 = 2.0 * eta * signb * sqb;
  double sx, cx;
  int iter = 0;
  while (iter < 20) {
    gamma2 = gamma1;
    gamma1 = gamma;
    double xx = 0.5 * gamma;
    if (beta0 > 0.0) {
      sincos_kepler(xx, &sx, &cx);
    } else {
      sx = sinh(xx);
      cx = exp(-xx) + sx;
    }
    gamma = gamma - (k * gamma + c2 * sx * cx + c3 * (sx * sx) + c4) /
                        (2.0 * signb * zeta * (sx * sx) + c5 * sx * cx + r0 * beta0);
    iter += 1;
    if (gamma == gamma2 || gamma == gamma1) break;
  }
  double xx = 0.5 * gamma;
  if (beta0 > 0.0) {
    sincos_kepler(xx, &sx, &cx);
  } else {
    sx = sinh(xx);
    cx = exp(-xx) + sx;
  }
  double g1bs = 2.0 * sx * cx / sqb;
  double g2bs = 2.0 * signb * (sx * sx) * beta0inv;
  double g0bs = 1.0 - beta0 * g2bs;
  constexpr int NEED = DRIFT_FIRST ? GH_G3 : (GH_G3 | GH_H1 | GH_H2);
  GH gh = gh_functions<NEED>(gamma, beta0, sqb);
  double g3bs = gh.g3;
  double h1 = 0.0, h2 = 0.0;
  double r = r0 * g0bs + eta * g1bs + k * g2bs;
  double rinv = 1.0 / r;
  double dfdt = (-k) * g1bs * rinv * r0inv;
  double fm1, gmh, dgdtm1;
  if (DRIFT_FIRST) {
    fm1 = (-k) * r0inv * g2bs;
    gmh = k * r0inv * (h * g2bs - r0 * g3bs);
    dgdtm1 = k * r0inv * rinv * (h * g1bs - r0 * g2bs);
  } else {
    h1 = gh.h1;
    h2 = gh.h2;
    fm1 = k * rinv * (g2bs - k * r0inv * h1);
    gmh = k * rinv * (r0 * h2 + eta * h1);
    dgdtm1 = (-k) * rinv * g2bs;
  }
  for (int j = 0; j < 3; j++) delxv[j] = fm1 * x0[j] + gmh * v0[j];
  for (int j = 0; j < 3; j++) delxv[3 + j] = dfdt * x0[j] + dgdtm1 * v0[j];
  P.gamma = gamma; P.g1 = g1bs; P.g2 = g2bs; P.g3 = g3bs;
  P.dfdt = dfdt; P.fm1 = fm1; P.gmh = gmh; P.dgdtm1 = dgdtm1; P.r0 = r0; P.r = r; P.r0inv = r0inv; P.rinv = rinv;
  P.k = k; P.h = h; P.beta = beta0; P.eta = eta; P.zeta = zeta;
}

// The Stumpff functions c_n(z) = sum_k (-z)^k / (n + 2k)!, n = 2..6, to degree
// 7 in -z: truncated below 2e-17 of c_n at |z| = KEP_ZMAX.
constexpr double KEP_ZMAX = 0.6;
__device__ constexpr double inv_factorial(int n) {
  double f = 1.0;
  for (int q = 2; q <= n; q++) f *= q;  // exact up to 18!, rounded once or twice beyond
  return 1.0 / f;
}
template <int NN>
__device__ __forceinline__ double stumpff(double z) {
  double p = inv_factorial(NN + 14);
#pragma unroll
  for (int k = 6; k >= 0; k--) p = fma(-z, p, inv_factorial(NN + 2 * k));
  return p;
}

// Derivatives of a solved drift (compute_jacobian_gamma!, ahl21.jl:896-1139,
// gives the same 6x8 block; here by the chain rule through s).
//
// With X = x0 - h v0 (drift first) or x0, V = v0, the drift is
// delx = A X + B V, delv = C X + D V, and A = k a(r0, eta, beta, k, h) and so
// on.  Kepler's equation gives ds by each of the five, dG_n = G_{n-1} ds +
// (n G_{n+2} - s G_{n+1}) / 2 dbeta, and r0, eta, beta depend on X, V through
// p = X.dX, V.dX + X.dV and w = V.dV alone:
//   dS = S[0] p + S[1] (V.dX + X.dV) + S[2] w + (k term) + S[4] dh,
// S[4] with x0 and v0 held.  S[3] is G k (dS/dk - S / k) / k, the part of the
// mass derivatives that does not cancel against the masses' own weights.
// About 150 FP64 instructions, a quarter of the expanded expressions'; the terms
// are sums of like sign or of different order in h, so none loses digits: K is
// off by 7.1e-16 rms of its 3x3 blocks (expanded: 8.9e-16), Psi by 8.6e-16
// (8.8e-16), the derivative by h by 3.7e-16 (4.0e-16), against binary128.
struct KepDeriv {
  double a[5], b[5], c[5], d[5];
};
template <bool DRIFT_FIRST, bool WITH_H>
__device__ __forceinline__ void kep_derivatives(const KepParams& P, KepDeriv& o) {
  const double r0 = P.r0, r0inv = P.r0inv, rinv = P.rinv, k = P.k;
  const double beta = P.beta, eta = P.eta, h = P.h, zeta = fma(-r0, beta, k);
  const double s = P.gamma * rsqrt_fast(fabs(beta));
  const double ss = s * s, z = beta * ss, s3 = ss * s, s4 = ss * ss;
  double g2, g3, g4, g5, g6;
  if (fabs(z) <= KEP_ZMAX) {
    const double c6 = stumpff<6>(z), c5 = stumpff<5>(z), c4 = fma(-z, c6, 1.0 / 24.0);
    g2 = ss * fma(-z, c4, 0.5);
    g3 = s3 * fma(-z, c5, 1.0 / 6.0);
    g4 = s4 * c4;
    g5 = (s4 * s) * c5;
    g6 = (s4 * ss) * c6;
  } else {
    const double bi = 1.0 / beta;
    g2 = P.g2;
    g3 = P.g3;
    g4 = (0.5 * ss - g2) * bi;
    g5 = (s3 * (1.0 / 6.0) - g3) * bi;
    g6 = (s4 * (1.0 / 24.0) - g4) * bi;
  }
  const double g1 = fma(-beta, g3, s);
  const double g0 = fma(-beta, g2, 1.0);
  const double h1 = fma(s, g3, -2.0 * g4), h2 = fma(s, g2, -g3);
  const double b1 = -0.5 * h2, b2 = -0.5 * h1, b3 = 0.5 * fma(3.0, g5, -(s * g4));  // dG_n / dbeta
  const double rp = fma(eta, g0, zeta * g1);                                        // dr / ds
  const double kr0 = k * r0inv;
  // s, and r at fixed s, by r0, eta, beta, k, h.  By k with beta = 2 k / r0 - v^2
  // moving along, so that zeta falls as k grows: its terms then differ in order
  // of h, where those at fixed beta and by beta would cancel to a fifth
  const double ri2 = 2.0 * r0inv, kb1 = ri2 * b1, kb2 = ri2 * b2, kb3 = ri2 * b3;
  const double ds[5] = {-(g1 * rinv), -(g2 * rinv), -(fma(k, b3, fma(eta, b2, r0 * b1)) * rinv),
                        fma(-zeta, kb3, fma(-eta, kb2, g3)) * rinv, rinv};
  const double rq[4] = {g0, g1, fma(-r0, g2, fma(eta, b1, zeta * b2)), fma(eta, kb1, fma(zeta, kb2, -g2))};
  constexpr int NQ = WITH_H ? 5 : 4;
  const double g2r = g2 * rinv, g1r = g1 * rinv, rr0 = r0inv * rinv;
  double al = 0.0, as = 0.0, bb = 0.0, bs = 0.0, hb1 = 0.0, hb2 = 0.0;
  if (!DRIFT_FIRST) {
    al = fma(-kr0, h1, g2) * rinv;           // A / k
    as = fma(-kr0, h2, g1);                  // by s, before the division by r
    bb = fma(eta, h1, r0 * h2) * rinv;       // B / k
    bs = fma(r0 * s, g1, eta * h2);
    hb1 = 0.5 * fma(5.0 * s, g5, fma(-ss, g4, -8.0 * g6));   // dH1 / dbeta
    hb2 = 0.5 * fma(3.0 * s, g4, fma(-ss, g3, -3.0 * g5));   // dH2 / dbeta
  }
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const double r_q = (q < 4) ? fma(rp, ds[q], rq[q]) : rp * ds[q];
    const double dg2 = (q == 2) ? fma(g1, ds[q], b2) : (q == 3) ? fma(g1, ds[q], kb2) : g1 * ds[q];
    const double dg1 = (q == 2) ? fma(g0, ds[q], b1) : (q == 3) ? fma(g0, ds[q], kb1) : g0 * ds[q];
    o.d[q] = rinv * fma(g2r, r_q, -dg2);
    o.c[q] = rr0 * fma(g1r, r_q, -dg1);
    if (q == 0) o.c[q] = fma(r0inv, g1r * r0inv, o.c[q]);
    if (DRIFT_FIRST) {
      o.a[q] = -(r0inv * dg2);
      if (q == 0) o.a[q] = fma(r0inv * r0inv, g2, o.a[q]);
      o.b[q] = (q == 2) ? fma(-g2, ds[q], -b3) : (q == 3) ? fma(-g2, ds[q], -kb3) : -(g2 * ds[q]);
    } else {
      double aq = as * ds[q], bq = bs * ds[q];
      if (q == 0) { aq = fma(kr0 * r0inv, h1, aq); bq = bq + h2; }
      if (q == 1) bq = bq + h1;
      if (q == 2) { aq = aq + fma(-kr0, hb1, b2); bq = bq + fma(r0, hb2, eta * hb1); }
      if (q == 3) {
        aq = aq + fma(-kr0 * ri2, hb1, fma(-r0inv, h1, kb2));
        bq = fma(ri2, fma(r0, hb2, eta * hb1), bq);
      }
      o.a[q] = rinv * fma(-al, r_q, aq);
      o.b[q] = rinv * fma(-bb, r_q, bq);
    }
  }
  const double kk = 2.0 * kr0 * r0inv * r0inv, gk = GNEWT * k, vv = fma(2.0, kr0, -beta);
  double* const f[4] = {o.a, o.b, o.c, o.d};
#pragma unroll
  for (int w = 0; w < 4; w++) {
    double* S = f[w];
    const double sb = S[2];
    S[0] = k * fma(-kk, sb, S[0] * r0inv);
    S[1] = k * S[1];
    S[2] = -2.0 * k * sb;
    S[3] = gk * S[3];
    if (WITH_H) S[4] = DRIFT_FIRST ? fma(k, S[4], -fma(eta, S[0], vv * S[1])) : k * S[4];
  }
  (void)h;
}

// The 6x6 block K of jac_kepler (row-major, rows delx, delv, columns x0, v0)
// and the mass vector Psi = G k d(delxv / k)/dk from the derivatives above.
template <bool DRIFT_FIRST>
__device__ __forceinline__ void kep_block(const KepParams& P, const KepDeriv& o, const double* x0, const double* v0,
                                          double* K, double* psi) {
  const double h = P.h;
  double X[3];
#pragma unroll
  for (int q = 0; q < 3; q++) X[q] = DRIFT_FIRST ? fma(-h, v0[q], x0[q]) : x0[q];
#pragma unroll
  for (int half = 0; half < 2; half++) {  // delx = A X + B V, then delv = C X + D V
    const double* U = half ? o.c : o.a;
    const double* W = half ? o.d : o.b;
    const double dx = half ? P.dfdt : P.fm1, dv = half ? P.dgdtm1 : P.gmh;
    double ux[3], wx[3], uv[3], wv[3];  // gradients by x0 and v0 of the two coefficients
#pragma unroll
    for (int q = 0; q < 3; q++) {
      ux[q] = fma(U[0], X[q], U[1] * v0[q]);
      wx[q] = fma(W[0], X[q], W[1] * v0[q]);
      uv[q] = fma(U[1], X[q], U[2] * v0[q]);
      wv[q] = fma(W[1], X[q], W[2] * v0[q]);
      if (DRIFT_FIRST) {
        uv[q] = fma(-h, ux[q], uv[q]);
        wv[q] = fma(-h, wx[q], wv[q]);
      }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double* row = K + 6 * (3 * half + i);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const double a = X[i] * ux[j], b = X[i] * uv[j];
        row[j] = fma(v0[i], wx[j], (i == j) ? a + dx : a);
        row[3 + j] = fma(v0[i], wv[j], (i == j) ? b + dv : b);
      }
      psi[3 * half + i] = fma(U[3], X[i], W[3] * v0[i]);
    }
  }
}

// d(delxv)/dh at fixed x0, v0 (the last column of jac_kepler).
template <bool DRIFT_FIRST>
__device__ __forceinline__ void kep_by_h(const KepParams& P, const KepDeriv& o, const double* x0, const double* v0,
                                         double* dh) {
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double X = DRIFT_FIRST ? fma(-P.h, v0[q], x0[q]) : x0[q];
    dh[q] = fma(o.a[4], X, o.b[4] * v0[q]);
    dh[3 + q] = fma(o.c[4], X, o.d[4] * v0[q]);
    if (DRIFT_FIRST) {
      dh[q] = fma(-P.fm1, v0[q], dh[q]);
      dh[3 + q] = fma(-P.dfdt, v0[q], dh[3 + q]);
    }
  }
}

}  // namespace nbg
