"""The cut-cell integrand without unneeded inverse cosines (CutCell) against
the full form (CellIntegrand): the same bits at every colatitude, over random
ceding and superseding regions (polar ones, nested and disjoint ones, azimuths
at and beyond half a turn, no superseding region), cells anywhere on the
circle, and colatitudes inside, across and outside both regions."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include "mesh_math.h"
#include <cstdio>
#include <cstring>
#include <random>
using namespace xgm;
int main() {
  std::mt19937_64 r(5);
  auto U = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(r); };
  long bad = 0, n = 0, lit = 0;
  for (int t = 0; t < 6000; t++) {
    const double colat = U(0.0, PI), rad = U(0.01, 1.5);
    double sc = 0.0, sr = 0.0, sa = 0.0;
    if (t % 4) {
      sc = U(0.0, PI); sr = U(0.005, 1.5);
      sa = t % 4 == 1 ? U(-0.5, 0.5) : (t % 4 == 2 ? U(-PI, PI) : U(-7.0, 7.0));
      if (t % 8 == 1) { sc = colat; sa = 0.0; }
    }
    const Region g = make_region(colat, rad, sr, sa, sc);
    const Star s{1.2e4, U(0.0, 0.2), U(0.1, 0.3), 0.0, 0};
    const double w = exp(U(log(1e-3), log(1.0)));
    double pa = U(-PI, PI - w), pb = pa + w;
    if (t % 16 == 0) { pa = -PI; pb = pa + w; }
    if (t % 16 == 8) { pb = PI + 1e-15; pa = pb - w; }
    if (t % 16 == 4) { pa = -0.5 * w; pb = 0.5 * w; }
    const CellIntegrand full{s, g, pa, pb};
    CutCell cut;
    const double lo = t % 2 ? 0.0 : fmax(0.0, colat - rad), hi = t % 2 ? PI : fmin(PI, colat + rad);
    cut.init(full, lo, hi);
    for (int k = 0; k <= 400; k++) {
      const double th = lo + (hi - lo) * (k / 400.0);
      const double a = full(th), b = cut(th);
      n++;
      lit += a != 0.0;
      if (std::memcmp(&a, &b, 8) != 0) bad++;
    }
    // a parallel's short range of colatitudes, as a cell's area integral sees it
    const double w1 = exp(U(log(1e-4), log(0.3))), l1 = U(0.0, PI - w1);
    cut.init(full, l1, l1 + w1);
    for (int k = 0; k <= 50; k++) {
      const double th = l1 + w1 * (k / 50.0);
      const double a = full(th), b = cut(th);
      n++;
      if (std::memcmp(&a, &b, 8) != 0) bad++;
    }
  }
  std::printf("%ld %ld %ld\n", bad, n, lit);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_cut_cell_bits(tmp_path):
    src = tmp_path / "cut.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "cut")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "xpsi_gb300", "csrc"), str(src), "-o", exe], check=True)
    bad, n, lit = map(int, subprocess.run([exe], check=True, capture_output=True,
                                          text=True).stdout.split())
    assert bad == 0
    assert lit > n // 20
