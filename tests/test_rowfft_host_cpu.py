"""The row transform's stages run on the host (fcb_rowfft.cuh outside nvcc): every shape, the even
(ramp) and the odd (Hilbert) kernel, against the direct sum in FP64."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "fastcone_b200", "csrc", "fcb_rowfft.cuh")

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "fcb_rowfft.cuh"
using namespace fcb::rf;

template <class S, bool ODD>
double error(int W)
{
  const int N = S::N, L = 2 * W;
  std::vector<double> h(W, 0.0), H(N + 1);
  for (int m = 0; m < W; m++) {
    if (ODD) h[m] = m % 2 ? 2.0 / (M_PI * m) : 0.0;
    else h[m] = m == 0 ? M_PI / 4 : m % 2 ? -1.0 / (M_PI * m * m) : 0.0;  // the ramp's kernel
  }
  for (int k = 0; k <= N; k++) {
    double a = ODD ? 0.0 : h[0];
    for (int m = 1; m < W; m++) {
      const double ph = M_PI * (double)((long long)k * m % (2 * N)) / N;
      a += ODD ? -2.0 * h[m] * sin(ph) : 2.0 * h[m] * cos(ph);
    }
    H[k] = a;
  }
  std::vector<cf> t1(S::T1), t2(S::T2 + 1), buf(S::BUF);
  std::vector<f4> g(S::G + 1);
  for (int i = 0; i < S::T1; i++) {
    const double ph = -2 * M_PI * ((i / S::BC) * (i % S::BC) % N) / N;
    t1[i] = {(float)cos(ph), (float)sin(ph)};
  }
  for (int i = 0; i < S::T2; i++) {
    const double ph = -2 * M_PI * ((i / S::C) * (i % S::C) % S::BC) / S::BC;
    t2[i] = {(float)cos(ph), (float)sin(ph)};
  }
  for (int i = 0; i <= S::G; i++) {
    const int k = entry_k<S>(i);
    g[i] = spectrum_entry(H[k], H[N - k], ODD, cos(M_PI * k / N), -sin(M_PI * k / N), N);
  }
  std::mt19937 r(W);
  std::normal_distribution<float> nd;
  std::vector<float> x(L), y(L, 0.0f);
  for (int i = 0; i < W; i++) x[i] = nd(r);
  auto pair = [&](int n) { return cf{2 * n < W ? x[2 * n] : 0.0f, 2 * n + 1 < W ? x[2 * n + 1] : 0.0f}; };
  for (int m = 0; m < S::NB1; m++) {
    cf v[S::HA];
    for (int a = 0; a < S::HA; a++) v[a] = pair(a * S::BC + m);
    stage1<S>(v, m, buf.data(), t1.data());
  }
  if constexpr (S::B > 1)
    for (int b = 0; b < S::NB2; b++) stage2<S, false>(b, buf.data(), t2.data());
  for (int q = 0; q < S::NB3; q++) stage3<S, ODD>(q, buf.data(), g.data());
  if constexpr (S::B > 1)
    for (int b = 0; b < S::NB2; b++) stage2<S, true>(b, buf.data(), t2.data());
  for (int m = 0; m < S::NB1; m++) {
    cf v[S::HA];
    stage1_back<S>(v, m, buf.data(), t1.data());
    for (int a = 0; a < S::HA; a++) {
      const int n = a * S::BC + m;
      if (2 * n < W) y[2 * n] = v[a].x;
      if (2 * n + 1 < W) y[2 * n + 1] = v[a].y;
    }
  }
  double e = 0.0, nrm = 0.0;
  for (int i = 0; i < W; i++) {
    double s = 0.0;
    for (int j = 0; j < W; j++) s += (ODD && j > i ? -1.0 : 1.0) * h[abs(i - j)] * x[j];
    e += (y[i] - s) * (y[i] - s);
    nrm += s * s;
  }
  return sqrt(e / nrm);
}

template <class S>
void shape()
{
  for (int W : {S::N, S::N - 1, S::N * 3 / 4 - 1}) printf("%d %d %d %d %.3e %.3e\n", S::A, S::B, S::C, W, error<S, false>(W), error<S, true>(W));
}

int main()
{
  @SHAPES@
}
"""


def test_every_shape_on_the_host(tmp_path):
    shapes = re.findall(r"Config<(Shape<\d+, \d+, \d+>)", open(HEADER).read())
    assert len(shapes) >= 15 and len(set(shapes)) == len(shapes)
    src = tmp_path / "rowfft.cpp"
    src.write_text(SOURCE.replace("@SHAPES@", "\n  ".join(f"shape<{s}>();" for s in shapes)))
    exe = str(tmp_path / "rowfft")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", os.path.dirname(HEADER), str(src), "-o", exe],
                   check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=120).stdout.split("\n")
    rows = [line.split() for line in out if line]
    assert len(rows) == 3 * len(shapes)
    for r in rows:
        # unit roundoff times the radix-2 depth of both transforms of the longest size, for white input
        assert float(r[4]) < 1.6e-6 and float(r[5]) < 1.6e-6, r
