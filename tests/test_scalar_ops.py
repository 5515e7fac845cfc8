"""The short forms of csrc/scalar_ops.h against the plain ones, on the host (the same IEEE arithmetic
as the device): the node search at interior nodes against the full 27-neighbour scan with its 0.99
rule -- on even and stretched lines, with the particle anywhere within two cells or many cells away along one axis, at midpoints
between nodes (where the rule decides) and on planes -- and the clamp against min and max, over
ordinary values, the bounds and their neighbours, zeros, infinities and NaN.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

SRC = r"""
#include "scalar_ops.h"
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>
#include <random>
using namespace cfd2lcs;
static const int NBR[27][3] = {
    {0, 0, 0},   {-1, 0, 0},  {0, -1, 0}, {0, 0, -1}, {1, 0, 0},  {0, 1, 0},  {0, 0, 1},   {-1, -1, -1}, {0, -1, -1},
    {1, -1, -1}, {-1, 0, -1}, {1, 0, -1}, {-1, 1, -1}, {0, 1, -1}, {1, 1, -1}, {-1, -1, 0}, {1, -1, 0},  {-1, 1, 0},
    {1, 1, 0},   {-1, -1, 1}, {0, -1, 1}, {1, -1, 1},  {-1, 0, 1}, {1, 0, 1},  {-1, 1, 1},  {0, 1, 1},   {1, 1, 1}};
template <class T> void full(const T q[3][3], int sa, int off[3]) {
  T best = 0;
  bool have = false;
  off[0] = off[1] = off[2] = 0;
  for (auto &o : NBR) {
    if (sa >= 0 && o[sa] != 0) continue;
    const T r = (q[0][o[0] + 1] + q[1][o[1] + 1]) + q[2][o[2] + 1];
    if (!have || r < T(0.99) * best) {
      best = r;
      have = true;
      for (int a = 0; a < 3; a++) off[a] = o[a];
    }
  }
}
template <class T> void search(long n, long &bad, long &moved, long &three) {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> U(0, 1);
  std::normal_distribution<double> N;
  for (long i = 0; i < n; i++) {
    T q[3][3];
    const int sa = i % 5 == 0 ? (int)(i / 5 % 3) : -1;
    const double mid = i % 3 == 0 ? 0.02 : (i % 3 == 1 ? 1e-9 : 1.0);  // how near to a midpoint
    for (int a = 0; a < 3; a++) {
      const double h0 = i % 2 ? 1.0 : 0.3 + U(g), h1 = i % 2 ? 1.0 : 0.3 + U(g);
      const double far = i % 7 == 0 && a == (int)(i % 3) ? 3 + 20 * U(g) : 0.0;  // many cells away along one axis
      const double at = far > 0 ? far : mid < 1 && U(g) < 0.7 ? (U(g) < 0.5 ? -0.5 * h0 : 0.5 * h1) + mid * N(g) : (U(g) * 4 - 2) * (U(g) < 0.5 ? 0.25 : 1.0);
      const T l[3] = {T(-h0), T(0), T(h1)}, x = T(at);
      for (int o = 0; o < 3; o++) {
        const T d = l[o] - x;
        q[a][o] = d * d;
      }
    }
    int u[3], v[3];
    full(q, sa, u);
    nbr_scan_short(q, sa, v);
    if (u[0] || u[1] || u[2]) moved++;
    if ((u[0] != 0) + (u[1] != 0) + (u[2] != 0) == 3) three++;
    if (u[0] != v[0] || u[1] != v[1] || u[2] != v[2]) bad++;
  }
}
int main() {
  long bad = 0, moved = 0, three = 0;
  search<double>(4000000, bad, moved, three);
  search<float>(4000000, bad, moved, three);
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  long cb = 0;
  auto clamp = [&](double v) { if (clamp01_select(v) != std::fmax(std::fmin(v, 1.0), 0.0)) cb++; };
  for (double v : {0.0, -0.0, 1.0, -1.0, 0.5, inf, -inf, nan, -nan, 1e-310, -1e-310, 1e300, -1e300, std::nextafter(1.0, 2.0), std::nextafter(1.0, 0.0),
                   std::nextafter(0.0, -1.0)})
    clamp(v);
  std::mt19937_64 g(7);
  std::normal_distribution<double> N;
  for (int i = 0; i < 2000000; i++) clamp(0.5 + N(g));
  printf("%ld %ld %ld %ld\n", bad, moved, three, cb);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_short_forms_equal_the_plain_ones(tmp_path):
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(SRC)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libcfd2lcs_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc, "-o", str(exe), str(src)], check=True)
    bad, moved, three, clamp = (int(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and clamp == 0
    assert moved > 1000000 and three > 100000  # moves along one axis and along all of them
