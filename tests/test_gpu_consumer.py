"""The Jacobian consumer's step on synthetic records, against an extended-precision consumer and the reference's sums.

column_step (csrc/nbg_jacobian.cuh) adds a step's increments to the compensation E and normalises the pair (S, E) where E
has grown, where the reference makes every update a Kahan sum (comp_sum_matrix!, src/utils.jl:36-46).  The probe runs
it on records of random Kepler blocks, masses, correctors and kicks, of the sizes they have in planetary systems, for
mass columns and others, with kick pairs and without.  The host applies the same records in long double (binary128 on
aarch64) and, as the reference does, by Kahan sums in double.  The bound is the reference's own error: over the columns
of a case, S + E is at most 1.25 times as far off, in the root mean square of each column's largest error over its
largest entry.  Without the compensation a column is ten times as far off, without the normalisation after the pairs
with body 0 one of eight bodies 1.33 times.
"""
import os
import subprocess
import tempfile

import pytest

from conftest import PKG_DIR, has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

PROBE = r'''
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "nbg_jacobian.cuh"
using namespace nbg;
typedef long double X;
constexpr int BS = 32;

template <int N, bool MASS, bool KICK>
__global__ void step(int R, int steps, double h, uint64_t kick, const double* rec, double* S, double* E) {
  __shared__ double sm[2 * 6 * N * BS];
  const int c0 = blockIdx.x * BS + threadIdx.x;  // a lane a column; the columns of the other kind idle
  const bool on = c0 < 7 * N && (c0 % 7 == 6) == MASS;
  double *s = sm + threadIdx.x, *e = sm + 6 * N * BS + threadIdx.x;
  if (!on) return;
  for (int r = 0; r < 6 * N; r++) s[r * BS] = S[r * 7 * N + c0], e[r * BS] = E[r * 7 * N + c0];
  for (int k = 0; k < steps; k++)
    column_step<N, BS, MASS, KICK>(s, e, c0, h, kick, Rec{const_cast<double*>(rec) + (size_t)k * R, 1});
  for (int r = 0; r < 6 * N; r++) S[r * 7 * N + c0] = s[r * BS], E[r * 7 * N + c0] = e[r * BS];
}

// The same step on a column of T, each update through add(row, increment)
template <int N, class T, class Get, class Add>
void host_step(int c, T h, uint64_t kick, const double* rec, Get get, Add add) {
  int off = 0;
  auto op = [&](const T* before, bool defer, std::vector<T>* out) {
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) {
        T acc = 0;
        for (int d = 0; d < N; d++)
          for (int p = 0; p < 3; p++) acc += (T)rec[off + (3 * b + k) * 4 * N + 4 * d + p] * before[6 * d + p];
        if (c % 7 == 6) acc += (T)rec[off + (3 * b + k) * 4 * N + 4 * (c / 7) + 3];
        if (defer) (*out)[3 * b + k] = acc;
        else add(6 * b + 3 + k, acc);
      }
    off += 12 * N * N;
  };
  std::vector<T> now(6 * N), k1(3 * N, (T)0);
  auto all = [&] { for (int r = 0; r < 6 * N; r++) now[r] = get(r); };
  auto drift = [&] {
    all();
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) add(6 * b + k, (h / 2) * now[6 * b + 3 + k]);
  };
  auto pair = [&](int i, int j) {
    const double* r = rec + off;
    all();
    T u[6];
    for (int a = 0; a < 6; a++) {
      u[a] = c % 7 == 6 && (c / 7 == i || c / 7 == j) ? (T)r[PREC_PSI + a] : (T)0;
      for (int l = 0; l < 6; l++) u[a] += (T)r[6 * a + l] * (now[6 * i + l] - now[6 * j + l]);
    }
    for (int a = 0; a < 6; a++) {
      add(6 * i + a, (T)r[PREC_MJ] * u[a] + (c == 7 * j + 6 ? (T)r[PREC_B + a] : (T)0));
      add(6 * j + a, -(T)r[PREC_MI] * u[a] - (c == 7 * i + 6 ? (T)r[PREC_B + a] : (T)0));
    }
    off += PREC;
  };
  if (kick) {  // formed before the drift, added after it (ahl21.jl:16-23)
    all();
    op(now.data(), true, &k1);
  }
  drift();
  if (kick)
    for (int b = 0; b < N; b++)
      for (int k = 0; k < 3; k++) add(6 * b + 3 + k, k1[3 * b + k]);
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++)
      if (!((kick >> pair_bit(i, j, N)) & 1)) pair(i, j);
  all();
  op(now.data(), false, nullptr);
  for (int i = N - 2; i >= 0; i--)
    for (int j = N - 1; j > i; j--)
      if (!((kick >> pair_bit(i, j, N)) & 1)) pair(i, j);
  drift();
  if (kick) {
    all();
    op(now.data(), false, nullptr);
  }
}

template <int N>
int run(bool kicks, int steps) {
  constexpr int M = 7 * N;
  std::mt19937_64 rng(100 * N + kicks);
  auto U = [&](double s) { return std::uniform_real_distribution<double>(-s, s)(rng); };
  uint64_t kick = 0;
  int npk = 0;
  for (int i = 0; i < N - 1; i++)
    for (int j = i + 1; j < N; j++) {
      if (kicks && i > 0) kick |= 1ull << pair_bit(i, j, N);
      else npk++;
    }
  const int R = step_record_size(N, npk, kick != 0);
  const double h = 0.5;
  std::vector<double> rec((size_t)steps * R);
  for (int k = 0; k < steps; k++) {
    double* r = &rec[(size_t)k * R];
    auto dense = [&] {  // an operator on position differences: its blocks over the bodies sum to zero
      for (int row = 0; row < 3 * N; row++) {
        for (int p = 0; p < 3; p++) {
          double sum = 0;
          for (int d = 1; d < N; d++) sum += (r[row * 4 * N + 4 * d + p] = std::ldexp(std::floor(U(1) * 65536), -36));
          r[row * 4 * N + p] = -sum;  // exact: few bits
        }
        for (int d = 0; d < N; d++) r[row * 4 * N + 4 * d + 3] = U(1e-6);
      }
      r += 12 * N * N;
    };
    auto pairs = [&](bool back) {
      for (int q = 0; q < N * (N - 1) / 2; q++) {
        const int at = back ? N * (N - 1) / 2 - 1 - q : q;
        if ((kick >> at) & 1) continue;
        const bool star = at < N - 1;
        const double n2 = star ? 4e-4 : 1e-9;  // G M / r^3 in 1/day^2
        for (int a = 0; a < 6; a++)
          for (int l = 0; l < 6; l++) r[6 * a + l] = U(1) * n2 * (a < 3 ? (l < 3 ? h * h : h * h * h) : (l < 3 ? h : h * h));
        const double m = star ? 1e-5 : 0.3;
        r[PREC_MI] = star ? 1 - m : m;
        r[PREC_MJ] = star ? m : 1 - m;
        for (int a = 0; a < 6; a++) r[PREC_PSI + a] = U(1e-5), r[PREC_B + a] = U(1e-4);
        r += PREC;
      }
    };
    if (kick) dense();
    pairs(false);
    dense();
    pairs(true);
    if (kick) dense();
  }
  std::vector<double> S0(6 * N * M), E0(6 * N * M);
  for (auto& v : S0) v = U(1);
  for (size_t q = 0; q < S0.size(); q++) E0[q] = U(1) * 5e-17 * std::fabs(S0[q]);
  double *dr, *dS, *dE;
  if (cudaMalloc(&dr, rec.size() * 8) || cudaMalloc(&dS, S0.size() * 8) || cudaMalloc(&dE, S0.size() * 8)) return 2;
  cudaMemcpy(dr, rec.data(), rec.size() * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(dS, S0.data(), S0.size() * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(dE, E0.data(), S0.size() * 8, cudaMemcpyHostToDevice);
  const int blocks = (M + BS - 1) / BS;
  if (kick) {
    step<N, false, true><<<blocks, BS>>>(R, steps, h, kick, dr, dS, dE);
    step<N, true, true><<<blocks, BS>>>(R, steps, h, kick, dr, dS, dE);
  } else {
    step<N, false, false><<<blocks, BS>>>(R, steps, h, 0, dr, dS, dE);
    step<N, true, false><<<blocks, BS>>>(R, steps, h, 0, dr, dS, dE);
  }
  std::vector<double> S(S0.size()), E(S0.size());
  if (cudaMemcpy(S.data(), dS, S.size() * 8, cudaMemcpyDeviceToHost) || cudaMemcpy(E.data(), dE, S.size() * 8, cudaMemcpyDeviceToHost))
    return 3;
  double ours = 0, theirs = 0;
  for (int c = 0; c < M; c++) {
    std::vector<X> x(6 * N);
    std::vector<double> s(6 * N), e(6 * N);
    for (int r = 0; r < 6 * N; r++) x[r] = (X)S0[r * M + c] + E0[r * M + c], s[r] = S0[r * M + c], e[r] = E0[r * M + c];
    for (int k = 0; k < steps; k++) {
      host_step<N, X>(c, h, kick, &rec[(size_t)k * R], [&](int r) { return x[r]; }, [&](int r, X a) { x[r] += a; });
      host_step<N, double>(c, h, kick, &rec[(size_t)k * R], [&](int r) { return s[r]; }, [&](int r, double a) {
        volatile double t0 = e[r] + a;
        volatile double t = s[r] + t0;
        volatile double d = s[r] - t;
        e[r] = d + t0;
        s[r] = t;
      });
    }
    X big = 0, a = 0, b = 0;
    for (int r = 0; r < 6 * N; r++) {
      big = std::max(big, fabsl(x[r]));
      a = std::max(a, fabsl((X)S[r * M + c] + E[r * M + c] - x[r]));
      b = std::max(b, fabsl((X)s[r] + e[r] - x[r]));
    }
    ours += (double)(a / big * a / big);
    theirs += (double)(b / big * b / big);
  }
  printf("%d %d %.6e %.6e\n", N, (int)kicks, std::sqrt(ours / M), std::sqrt(theirs / M));
  return 0;
}
int main() {
  const int steps = 2000;
  return run<2>(false, steps) | run<3>(false, steps) | run<8>(false, steps) | run<3>(true, steps) | run<5>(true, steps);
}
'''


def test_column_step_against_long_double_and_kahan_sums():
    with tempfile.TemporaryDirectory() as tmp:
        src, exe = os.path.join(tmp, "c.cu"), os.path.join(tmp, "c")
        with open(src, "w") as f:
            f.write(PROBE)
        subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                        "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(PKG_DIR, "csrc"), "-o", exe, src], check=True)
        out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == 5
    for line in out:
        n, kicks, ours, theirs = line.split()
        assert float(ours) <= 1.25 * float(theirs), line
