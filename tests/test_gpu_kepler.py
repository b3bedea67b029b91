"""The Kepler drift of a pair and its derivatives against an extended-precision oracle.

kep_solve, kep_derivatives, kep_block and kep_by_h (csrc/nbg_kepler.cuh) run on seeded pairs; the oracle solves the same
drift in universal variables with numpy's long double (binary128 on the GPU's aarch64 hosts, 80 bits on x86) on dual
numbers, so that the 6x6 block K, Psi = G k d(delxv / k)/dk and the derivative by the step come without differences.

Bounds, set from what the reference's expanded expressions (ahl21.jl:896-1139) leave in double precision on the same
draws: rms over a class K 8.9e-16 of its 3x3 blocks, Psi 8.8e-16, by h 4.4e-16, delxv 4.2e-16, a tenth more for the
draw, a third more for planet pairs' Psi; single values at most 8 rms.  Eccentric and long steps have wider rms bounds and
none on single values: there the drift's end hangs on the start's last digits, by factors that differ from pair to pair
(delxv itself, whose rounding is the reference's, is 1.4e-14 off at worst).
"""
import os
import subprocess
import tempfile

import numpy as np
import pytest

from conftest import PKG_DIR, has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

GNEWT = 39.4845 / (365.242 * 365.242)
LD = np.longdouble

PROBE = r'''
#include <cstdio>
#include <vector>
#include "nbg_kepler.cuh"
using namespace nbg;
constexpr int IN = 9, OUT = 54;
template <bool DF> __device__ void one(const double* in, double* out) {
  const double k = GNEWT * (in[6] + in[7]);
  KepParams P;
  KepDeriv D;
  kep_solve<DF>(in, in + 3, k, in[8], out, P);
  kep_derivatives<DF, true>(P, D);
  kep_block<DF>(P, D, in, in + 3, out + 6, out + 42);
  kep_by_h<DF>(P, D, in, in + 3, out + 48);
}
__global__ void run(int n, const double* in, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double a[IN], b[OUT];
  for (int q = 0; q < IN; q++) a[q] = in[(size_t)t * IN + q];
  one<true>(a, b);
  for (int q = 0; q < OUT; q++) out[(size_t)t * 2 * OUT + q] = b[q];
  one<false>(a, b);
  for (int q = 0; q < OUT; q++) out[(size_t)t * 2 * OUT + OUT + q] = b[q];
}
int main(int argc, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  int n = 0;
  if (!f || fread(&n, sizeof(int), 1, f) != 1 || n <= 0 || n > (1 << 20)) return 2;
  std::vector<double> in((size_t)n * IN), out((size_t)n * 2 * OUT);
  if (fread(in.data(), 8, in.size(), f) != in.size()) return 3;
  fclose(f);
  double *di, *dout;
  if (cudaMalloc(&di, in.size() * 8) != cudaSuccess || cudaMalloc(&dout, out.size() * 8) != cudaSuccess) return 4;
  cudaMemcpy(di, in.data(), in.size() * 8, cudaMemcpyHostToDevice);
  run<<<(n + 127) / 128, 128>>>(n, di, dout);
  if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 5;
  f = fopen(argv[2], "wb");
  fwrite(out.data(), 8, out.size(), f);
  fclose(f);
  return 0;
}
'''


# ------------------------------------------------------------------ the oracle: dual numbers, [value, d/dx, d/dv, d/dk, d/dh]

def mul(a, b):
    r = a * b[:1] + a[:1] * b
    r[0] = a[0] * b[0]
    return r


def func(a, value, slope):
    r = a * slope
    r[0] = value
    return r


def inv(a):
    return func(a, 1 / a[0], -1 / a[0] ** 2)


def root(a):
    v = np.sqrt(a[0])
    return func(a, v, 1 / (2 * v))


def dot(a, b):
    return sum(mul(p, q) for p, q in zip(a, b))


def stumpff(n, z):
    """c_n(z) and its derivative by z."""
    term = LD(1) / LD(int(np.prod(np.arange(2, n + 1))))
    c, d = np.zeros_like(z), np.zeros_like(z)
    power, before = np.ones_like(z), np.zeros_like(z)
    for k in range(40):
        c = c + term * power
        d = d + term * k * before
        before = power
        power = power * z
        term = -term / LD((n + 2 * k + 1) * (n + 2 * k + 2))
    return c, d


def drift(x, v, k, h, drift_first):
    """delxv / k as duals, from duals; values and derivatives of each step in long double."""
    X = [p - mul(h, q) for p, q in zip(x, v)] if drift_first else list(x)
    r0 = root(dot(X, X))
    r0i = inv(r0)
    eta, vv = dot(X, v), dot(v, v)
    beta = 2 * mul(k, r0i) - vv
    zeta = k - mul(r0, beta)
    s = h[0] * r0i[0]
    for _ in range(60):
        z = beta[0] * s * s
        g2, g3 = s * s * stumpff(2, z)[0], s ** 3 * stumpff(3, z)[0]
        r = r0[0] + eta[0] * (s - beta[0] * g3) + zeta[0] * g2
        s = s - (r0[0] * s + eta[0] * g2 + zeta[0] * g3 - h[0]) / r

    def functions(sd):
        ss = mul(sd, sd)
        z = mul(beta, ss)
        g2, g3 = mul(ss, func(z, *stumpff(2, z[0]))), mul(mul(ss, sd), func(z, *stumpff(3, z[0])))
        g1 = sd - mul(beta, g3)
        return g1, g2, g3, r0 + mul(eta, g1) + mul(zeta, g2)

    fixed = np.zeros_like(r0)
    fixed[0] = s
    _, g2, g3, r = functions(fixed)
    step = mul(mul(r0, fixed) + mul(eta, g2) + mul(zeta, g3) - h, inv(func(r * 0, r[0], 0)))
    step[0] = 0
    g1, g2, g3, r = functions(fixed - step)
    ri = inv(r)
    f, fd, gd = -mul(r0i, g2), -mul(mul(r0i, ri), g1), -mul(ri, g2)
    dv = [mul(fd, p) + mul(gd, q) for p, q in zip(X, v)]
    dx = [mul(f, p) - mul(g3, q) for p, q in zip(X, v)]
    if not drift_first:
        dx = [p - mul(h, q) for p, q in zip(dx, dv)]
    return dx + dv


def oracle(pairs, drift_first):
    n = len(pairs)
    dual = np.zeros((8, 9, n), dtype=LD)
    for q in range(6):
        dual[q, 0] = pairs[:, q]
    dual[6, 0] = GNEWT * (pairs[:, 6] + pairs[:, 7])  # rounded as the device's
    dual[7, 0] = pairs[:, 8]
    for q in range(8):
        dual[q, 1 + q] = 1
    out = dual[6, 0] * np.array(drift(list(dual[:3]), list(dual[3:6]), dual[6], dual[7], drift_first))  # [6][9][n]
    return out[:, 0], out[:, 1:7], LD(GNEWT) * out[:, 7], out[:, 8]  # by k: k d(delxv / k)/dk


def star_pairs(rng, n, e, part):
    """Star-planet pairs of a period of 1 to 100 days, a step of `part` of it; x, v, m_i, m_j, h."""
    P, m = np.exp(rng.uniform(0, np.log(100), n)), np.exp(rng.uniform(np.log(1e-6), np.log(1e-4), n))
    ecc, M = rng.uniform(*e, n), rng.uniform(0, 2 * np.pi, n)
    k = GNEWT * (1 + m)
    E = M.copy()
    for _ in range(100):
        E = E - (E - ecc * np.sin(E) - M) / (1 - ecc * np.cos(E))
    a, w = np.cbrt(k * P * P / (4 * np.pi ** 2)), rng.uniform(0, 2 * np.pi, n)
    tilt = np.pi / 2 + rng.uniform(-0.02, 0.02, n)
    b, nu = np.sqrt(1 - ecc ** 2), 2 * np.pi / P / (1 - ecc * np.cos(E))
    px, py, vx, vy = a * (np.cos(E) - ecc), a * b * np.sin(E), -a * nu * np.sin(E), a * nu * b * np.cos(E)
    turn = lambda p, q: (np.cos(w) * p - np.sin(w) * q, np.sin(w) * p + np.cos(w) * q)  # noqa: E731
    (x, y), (u, t) = turn(px, py), turn(vx, vy)
    h = part * P * np.where(rng.random(n) < 0.1, -1, 1)
    return np.stack([x, y * np.cos(tilt), y * np.sin(tilt), u, t * np.cos(tilt), t * np.sin(tilt), np.ones(n), m, h], 1)


def planet_pairs(rng, n):
    """Unbound pairs of planets."""
    m = np.exp(rng.uniform(np.log(1e-6), np.log(1e-4), (n, 2)))
    return np.hstack([rng.uniform(-0.3, 0.3, (n, 3)), rng.uniform(-0.08, 0.08, (n, 3)), m, rng.uniform(0.03, 0.3, (n, 1))])


COUNT = 2000
STAR = {"delxv": 4.7e-16, "K": 9.8e-16, "psi": 9.7e-16, "h": 4.9e-16}
# class: pairs, and the rms bound of each quantity by drift order (None: not bounded)
CLASSES = {
    "bound": (lambda r: star_pairs(r, COUNT, (0, 0.3), 0.025 * r.uniform(0.02, 1, COUNT)), STAR, STAR),
    "planets": (lambda r: planet_pairs(r, COUNT), {**STAR, "psi": 1.2e-15}, {**STAR, "psi": 1.2e-15}),
    # e up to 0.95: half steps of a fortieth of the period
    "eccentric": (lambda r: star_pairs(r, COUNT, (0.8, 0.95), 0.025), None,
                  {"delxv": 2e-15, "K": 1e-14, "psi": 2e-14, "h": 2e-15}),
    # beta s^2 on both sides of KEP_ZMAX
    "long": (lambda r: star_pairs(r, COUNT, (0, 0.3), r.uniform(0.1, 0.16, COUNT)), None,
             {"delxv": 1e-15, "K": 4e-15, "psi": 1e-14, "h": 1e-15}),
}


@pytest.fixture(scope="module")
def device():
    """Runs the probe on an array of pairs: [n][2][54]."""
    with tempfile.TemporaryDirectory() as tmp:
        src, exe = os.path.join(tmp, "k.cu"), os.path.join(tmp, "k")
        with open(src, "w") as f:
            f.write(PROBE)
        subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
                        "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)

        def go(pairs):
            a, b = os.path.join(tmp, "in"), os.path.join(tmp, "out")
            with open(a, "wb") as f:
                f.write(np.int32(len(pairs)).tobytes())
                f.write(np.ascontiguousarray(pairs, dtype=np.float64).tobytes())
            subprocess.run([exe, a, b], check=True)
            return np.fromfile(b).reshape(len(pairs), 2, 54)

        yield go


def norms(a):
    """Over the vector's position and velocity halves, [6][n] -> [2][n]."""
    return np.sqrt((a.reshape(2, 3, -1) ** 2).sum(1))


def compare(got, pairs, drift_first):
    """Relative errors of each quantity, the larger of its halves or blocks, per pair."""
    delxv, K, psi, by_h = oracle(pairs, drift_first)
    half = lambda g, r: (norms(g.T.astype(LD) - r) / norms(r)).max(0)  # noqa: E731
    block = lambda a: np.sqrt((a.reshape(2, 3, 2, 3, -1) ** 2).sum((1, 3)))  # noqa: E731
    k = got[:, 6:42].reshape(-1, 6, 6).transpose(1, 2, 0).astype(LD)
    return {"delxv": half(got[:, :6], delxv), "K": (block(k - K) / block(K)).max((0, 1)),
            "psi": half(got[:, 42:48], psi), "h": half(got[:, 48:54], by_h)}


@pytest.mark.parametrize("drift_first", [True, False])
@pytest.mark.parametrize("name", list(CLASSES))
def test_drift_and_derivatives(device, name, drift_first):
    make, first, last = CLASSES[name]
    bounds = first if drift_first else last
    if bounds is None:
        pytest.skip("a step past the pericentre or over a sixth of an orbit is ill-conditioned with the drift first")
    pairs = make(np.random.default_rng(17))
    err = compare(device(pairs)[:, 0 if drift_first else 1], pairs, drift_first)
    for q, bound in bounds.items():
        rms = float(np.sqrt((err[q] ** 2).mean()))
        assert rms <= bound, (q, rms)
        if name in ("bound", "planets"):
            assert float(err[q].max()) <= 8 * bound, (q, float(err[q].max()))


ELEMENTARY = r'''
#include <cstdio>
#include <vector>
#include "nbg_kepler.cuh"
using namespace nbg;
__global__ void run(int n, const double* x, const double* z, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double* o = out + (size_t)t * 7;
  o[0] = rcp_fast(x[t]);
  o[1] = rsqrt_fast(fabs(x[t]));
  o[2] = stumpff<2>(z[t]);
  o[3] = stumpff<3>(z[t]);
  o[4] = stumpff<4>(z[t]);
  o[5] = stumpff<5>(z[t]);
  o[6] = stumpff<6>(z[t]);
}
int main(int argc, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  int n = 0;
  if (!f || fread(&n, sizeof(int), 1, f) != 1 || n <= 0 || n > (1 << 22)) return 2;
  std::vector<double> in((size_t)n * 2), out((size_t)n * 7);
  if (fread(in.data(), 8, in.size(), f) != in.size()) return 3;
  fclose(f);
  double *di, *dout;
  if (cudaMalloc(&di, in.size() * 8) != cudaSuccess || cudaMalloc(&dout, out.size() * 8) != cudaSuccess) return 4;
  cudaMemcpy(di, in.data(), in.size() * 8, cudaMemcpyHostToDevice);
  run<<<(n + 127) / 128, 128>>>(n, di, di + n, dout);
  if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 5;
  f = fopen(argv[2], "wb");
  fwrite(out.data(), 8, out.size(), f);
  fclose(f);
  return 0;
}
'''


def test_reciprocal_root_and_stumpff_sums():
    """rcp_fast and rsqrt_fast over 2^-300 to 2^300 and the Stumpff sums over |z| <= KEP_ZMAX, against long double.

    u = 2^-53.  rcp_fast: the last FMA's rounding, u, and e's own error times the seed's (below u / 1000).  rsqrt_fast:
    that and half of the rounding of x y, which e carries whole: 1.5 u.  stumpff: the last sum's rounding and its
    coefficient's, 2 u, and z c_{n+2} / c_n <= 0.05 of as much again, and the truncation, below 0.2 u."""
    rng, n = np.random.default_rng(5), 1 << 17
    x = np.exp2(rng.uniform(-300, 300, n)) * rng.choice([-1.0, 1.0], n)
    z = rng.uniform(-0.6, 0.6, n)
    z[:3] = 0.0, 0.6, -0.6
    with tempfile.TemporaryDirectory() as tmp:
        src, exe, a, b = (os.path.join(tmp, q) for q in ("e.cu", "e", "in", "out"))
        with open(src, "w") as f:
            f.write(ELEMENTARY)
        subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
                        "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)
        with open(a, "wb") as f:
            f.write(np.int32(n).tobytes() + x.tobytes() + z.tobytes())
        subprocess.run([exe, a, b], check=True)
        got = np.fromfile(b).reshape(n, 7).astype(LD)
    u = LD(2) ** -53
    off = lambda g, r: float((np.abs(g - r) / np.abs(r)).max() / u)  # noqa: E731
    assert off(got[:, 0], 1 / x.astype(LD)) <= 1.01
    assert off(got[:, 1], 1 / np.sqrt(np.abs(x).astype(LD))) <= 1.51
    for k in range(2, 7):
        assert off(got[:, k], stumpff(k, z.astype(LD))[0]) <= 2.4, k
