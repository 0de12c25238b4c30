"""The height of the pruned mixed form, on the host: the library's height where
it has the form, else a taller one only within the limits where it measured
faster, so that no call pays for a much taller grid.  Calls: at most 1.2 times as
tall with the stored columns at most 0.6 of the library's row, or 1.1 times and
0.8; grids that plans and streams keep: 1.5 times and 0.7, or 1.2 times and 0.8;
any height up to 1024 rows.
"""
import os
import subprocess

import pytest

from wsclean_b200.gridder import plan_grid

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wsclean_b200", "csrc")
PX = 1e-5


@pytest.mark.parametrize("n,v,most", [(1516, 0.34, 2592), (3148, 0.36, 5376), (5796, 0.20, 10000)])
def test_taller_grids_that_cost_more_are_left(n, v, most):
    assert plan_grid(n, n, PX, PX, 1e-5, 10 ** 6, 0.0, 200.0, v / PX)["nv"] <= most


@pytest.mark.parametrize("n,v,nv", [(4096, 0.145, 6144), (8192, 0.208, 16384)])
def test_taller_grids_that_pay_are_taken(n, v, nv):
    assert plan_grid(n, n, PX, PX, 1e-5, 10 ** 6, 0.0, 200.0, v / PX)["nv"] == nv


PROGRAM = r'''
#include <cstdio>
#include "wsg_internal.h"

int main() {
  long higher = 0, natural = 0, whole = 0, wrong = 0;
  for (bool resident : {false, true})
   for (double eps : {1e-4, 1e-5})
    for (int n = 200; n < 9000; n += 2 * (1 + n / 40))
      for (double v : {0.05, 0.12, 0.2, 0.28, 0.36, 0.45}) {
        wsg::GridPlan g;
        g.nx = g.ny = size_t(n);
        g.px = g.py = 1e-5;
        g.eps = eps;
        g.do_w = true;
        g.fp32 = true;
        g.nvis = 1000000;
        g.wmax_d = 200;
        g.umax = g.vmax = v / g.px;
        g.resident = resident;
        wsg::GridPlan w = g;
        w.whole_rows = true;
        wsg::choose_grid(g, 1.1, 2.0, 24);
        wsg::choose_grid(w, 1.1, 2.0, 24);
        if (w.vprune || g.nplanes != w.nplanes || g.nu != w.nu) ++wrong;
        if (!g.vprune) {
          ++whole;
          if (g.nv != w.nv) ++wrong;
        } else if (g.nv == w.nv) {
          ++natural;
        } else {
          ++higher;
          const double taller = double(g.nv) / w.nv, stored = (double(g.nvs()) - 1) / w.nv;
          auto within = [&](double t, double c) { return taller <= t && stored <= c; };
          const bool pays = g.nv <= 1024 || (resident ? within(1.5, 0.7) || within(1.2, 0.8)
                                                      : within(1.2, 0.6) || within(1.1, 0.8));
          if (!pays || g.kernel.err > 1.05e-5) ++wrong;
        }
      }
  std::printf("%ld %ld %ld %ld\n", wrong, higher, natural, whole);
  return 0;
}
'''


def test_limits_over_sizes(tmp_path):
    src = tmp_path / "heights.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "heights"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    str(src), os.path.join(CSRC, "es_kernel.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    wrong, higher, natural, whole = (int(x) for x in out.split())
    assert higher > 20 and natural > 20 and whole > 20, out
    assert wrong == 0, out
