"""Rounding of the mixed-radix transforms (csrc/fft_mx.cuh), on the CPU: the
header's twiddle tables and butterflies, compiled for the host and run."""
from __future__ import annotations

import importlib.util
import os
import subprocess

from conftest import PKG_DIR

HEAD = r"""
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>
#include "fft_mx.cuh"
using namespace gila;
using Line = std::vector<double2>;
using Exact = std::complex<long double>;
constexpr long double kPi = 3.14159265358979323846264338327950288L;

template <typename W> W unit(int P, int m);  // exp(-2 pi i m / P), rounded once
template <> double2 unit<double2>(int P, int m) {
  const long double a = -2.0L * kPi * (long double)m / (long double)P;
  return double2{(double)cosl(a), (double)sinl(a)};
}
template <> float2 unit<float2>(int P, int m) {
  const double2 d = unit<double2>(P, m);
  return float2{(float)d.x, (float)d.y};
}
template <typename W> std::vector<W> table(int P) {
  std::vector<W> tab(mx_tw_len(P));
  for (int m = 0; m < P; ++m) tab[m] = unit<W>(P, m);
  mx_tw_fill(P, [&](int at, int m) { tab[at] = tab[m]; });
  return tab;
}
"""

FACTORS = HEAD + r"""
static long bad = 0, seen = 0;
template <typename W, int P, int KIND, bool REV, bool INV, int S> void stage(const std::vector<W>& tab) {
  constexpr int R = mx_r<P, KIND, REV>(S), NS = mx_span<P, KIND, REV>(S);
  for (int jm = 0; jm < NS; ++jm) {
    W w[R];
    mx_twiddles<R, NS, INV>(tab.data() + MxTw<P, KIND, REV, S>::off + jm, w);
    for (int q = 1; q < R; ++q) {
      W e = unit<W>(P, (int)((long)q * jm * (P / (NS * R)) % P));
      if (INV) e.y = -e.y;
      ++seen;
      bad += !(w[q].x == e.x && w[q].y == e.y);
    }
  }
  if constexpr (S + 1 < MxPlan<P, KIND>::s.n) stage<W, P, KIND, REV, INV, S + 1>(tab);
}
template <typename W, int P> void length() {
  const std::vector<W> tab = table<W>(P);
  if constexpr (MxPlan<P, MXK_XY>::s.n > 1) {
    stage<W, P, MXK_XY, false, false, 1>(tab);
    stage<W, P, MXK_XY, false, true, 1>(tab);
  }
  if constexpr (MxPlan<P, MXK_Z>::s.n > 1) {
    stage<W, P, MXK_Z, false, false, 1>(tab);
    stage<W, P, MXK_Z, true, true, 1>(tab);
  }
}
template <int... P> void all() { (length<double2, P>(), ...); (length<float2, P>(), ...); }
int main() {
  all<12, 20, 28, 32, 36, 54, 72, 96, 100, 120, 162, 168, 210, 240, 250, 300, 384, 392, 500, 504>();
  printf("%ld %ld\n", bad, seen);
}
"""

# rms error of a forward transform of a half-filled line and of an inverse one:
# the length's x / y and z plans, and the plan of the runtime-planned kernels
# (factors 8, then 4 or 2, 3, 5, 7, every twiddle rounded once)
ERRORS = HEAD + r"""
template <bool INV> void dft(int R, double2* v) {
  switch (R) {
    case 2: Dft<2, INV>::run(v); break;
    case 3: Dft<3, INV>::run(v); break;
    case 4: Dft<4, INV>::run(v); break;
    case 5: Dft<5, INV>::run(v); break;
    case 7: Dft<7, INV>::run(v); break;
    case 8: Dft<8, INV>::run(v); break;
  }
}
template <bool INV> Line general(const Line& x) {
  const int P = (int)x.size();
  std::vector<int> rad;
  int n = P, twos = 0;
  for (; n % 2 == 0; n /= 2) ++twos;
  for (; twos >= 3; twos -= 3) rad.push_back(8);
  if (twos) rad.push_back(1 << twos);
  for (int q : {3, 5, 7})
    for (; n % q == 0; n /= q) rad.push_back(q);
  Line a = x, b(P);
  int ns = 1;
  for (int R : rad) {
    const int T = P / R, st = P / (ns * R);
    for (int j = 0; j < T; ++j) {
      const int jm = j % ns;
      double2 v[8], w[8];
      auto tw = [&](long m) {
        double2 u = unit<double2>(P, (int)(m % P));
        if (INV) u.y = -u.y;
        return u;
      };
      for (int r = 1; r < R; ++r) w[r] = tw((long)r * jm * st);
      for (int r = 0; r < R; ++r) v[r] = r && ns > 1 ? vmul(a[j + r * T], w[r]) : a[j + r * T];
      dft<INV>(R, v);
      for (int r = 0; r < R; ++r) b[(j - jm) * R + jm + r * ns] = v[r];
    }
    std::swap(a, b);
    ns *= R;
  }
  return a;
}
template <int P, int KIND, bool REV, bool INV, int S> void stages(const std::vector<double2>& tab, Line& a) {
  constexpr int R = mx_r<P, KIND, REV>(S), NS = mx_span<P, KIND, REV>(S), T = P / R;
  Line b(P);
  for (int j = 0; j < T; ++j) {
    const int jm = j % NS;
    double2 v[R], w[R];
    if constexpr (NS > 1) mx_twiddles<R, NS, INV>(tab.data() + MxTw<P, KIND, REV, S>::off + jm, w);
    for (int r = 0; r < R; ++r) v[r] = r && NS > 1 ? vmul(a[j + r * T], w[r]) : a[j + r * T];
    Dft<R, INV>::run(v);
    for (int r = 0; r < R; ++r) b[(j - jm) * R + jm + r * NS] = v[r];
  }
  a = b;
  if constexpr (S + 1 < MxPlan<P, KIND>::s.n) stages<P, KIND, REV, INV, S + 1>(tab, a);
}
template <typename F, typename I> double error(int P, const F& fwd, const I& inv) {
  std::mt19937_64 g(5);
  std::normal_distribution<double> N;
  std::vector<Exact> W(P);
  for (int m = 0; m < P; ++m) W[m] = std::polar(1.0L, -2.0L * kPi * m / P);
  double d[2] = {0, 0}, n[2] = {0, 0};
  for (int k = 0; k < std::max(4, 8000 / P); ++k)
    for (int dir = 0; dir < 2; ++dir) {
      const int from = dir ? P : P / 2, to = dir ? P / 2 : P;
      Line x(P, double2{0.0, 0.0});
      for (int i = 0; i < from; ++i) x[i] = double2{N(g), N(g)};
      const Line y = dir ? inv(x) : fwd(x);
      for (int q = 0; q < to; ++q) {
        Exact s = 0;
        for (int i = 0; i < from; ++i) s += (dir ? std::conj(W[(long)q * i % P]) : W[(long)q * i % P]) * Exact(x[i].x, x[i].y);
        d[dir] += (double)std::norm(s - Exact(y[q].x, y[q].y));
        n[dir] += (double)std::norm(s);
      }
    }
  return std::sqrt(d[0] / n[0] + d[1] / n[1]);
}
template <int P> void length() {
  const std::vector<double2> tab = table<double2>(P);
  const double g = error(P, general<false>, general<true>);
  const double xy = error(P, [&](Line x) { stages<P, MXK_XY, false, false, 0>(tab, x); return x; },
                          [&](Line x) { stages<P, MXK_XY, false, true, 0>(tab, x); return x; });
  const double z = error(P, [&](Line x) { stages<P, MXK_Z, false, false, 0>(tab, x); return x; },
                         [&](Line x) { stages<P, MXK_Z, true, true, 0>(tab, x); return x; });
  printf("%d %.17g %.17g %.17g\n", P, g, xy, z);
}
template <int... P> void all() { (length<P>(), ...); }
int main() { all<16, 24, 28, 36, 48, 60, 72, 84, 100, 120, 168, 180, 240, 300>(); }
"""


def _build_module():
    spec = importlib.util.spec_from_file_location("gila_build", os.path.join(PKG_DIR, "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def _run(program, tmp_path):
    b = _build_module()
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(program)
    # fused multiply-adds only where the source asks for them
    subprocess.run([b._nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-mfma,-ffp-contract=off", "-I", b.CSRC, str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout


def test_stage_twiddles_are_rounded_once(tmp_path):
    """Every factor that a stage multiplies by is the exact value rounded
    once: a factor formed as a product of others carries their roundings into
    the spectrum."""
    bad, seen = (int(v) for v in _run(FACTORS, tmp_path).split())
    assert seen > 10000 and bad == 0


def test_rounding_no_larger_than_the_runtime_plan(tmp_path):
    """A product transforms two axes by the x / y plan and one by the z plan:
    over the three, the rms error of no length exceeds that of the general
    kernels' plan.  The errors are rms values of 8000 elements or more a
    direction, whose statistical deviation is below 1 %; the bound allows two
    of them."""
    for line in _run(ERRORS, tmp_path).splitlines():
        P, g, xy, z = (float(v) for v in line.split())
        assert (2 * xy ** 2 + z ** 2) ** 0.5 <= 1.02 * (3 * g ** 2) ** 0.5, (P, g, xy, z)
