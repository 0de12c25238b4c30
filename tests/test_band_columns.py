"""The stored columns of the band grid (``band_col`` / ``band_col_next`` of
``wsg_internal.h``), on the host over planned grids: from every cell of every
tile a line may start at, each cell of the longest line falls on the column of
its v, or outside the row when v is outside the band -- also where a tile holds
both ends of a band nearly as wide as the grid, or is longer than the grid."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wsclean_b200", "csrc")

PROGRAM = r'''
#include <algorithm>
#include <cstdio>
#include "wsg_internal.h"

int main() {
  long wrong = 0, pruned = 0, both = 0, whole = 0, small = 0;
  for (double eps : {1e-3, 1e-4, 1e-5})
    for (int ny : {2, 4, 6, 8, 10, 12, 16, 18, 20, 22, 24, 28, 32, 40, 50, 64, 128, 136, 150,
                   160, 170, 180, 250, 276, 300, 340, 360, 512, 560, 640, 680, 720, 1024, 1118, 2048})
      for (double vpx : {0.1, 0.3, 0.4, 0.46, 0.465, 0.47, 0.48, 0.488, 0.492, 0.494, 0.498}) {
        wsg::GridPlan g;
        g.nx = 64;
        g.ny = size_t(ny);
        g.px = g.py = 0.08 / 256;
        g.eps = eps;
        g.do_w = true;
        g.fp32 = true;
        g.nvis = 100000;
        g.wmin_d = 0;
        g.wmax_d = 10;
        g.umax = 0.2 / g.px;
        g.vmax = vpx / g.py;
        try {
          wsg::choose_grid(g, 1.1, 2.0, 24);
        } catch (const wsg::InvalidArgument &) {
          continue;  // (images smaller than the kernel)
        }
        const int nv = int(g.nv), nvs = int(g.nvs()), Lv = g.vprune ? int(g.Lv) : 0;
        const int n = g.T + g.kernel.W - 1;  // cells along v of a tile
        (g.vprune ? pruned : whole) += 1;
        if (g.vprune && nv - 2 * Lv - 1 < n) ++both;
        if (nv < n) ++small;
        for (int tv = 0; tv < g.ntv; ++tv)
          for (int ib = 0; ib < n; ++ib) {
            int v0 = tv * g.T - g.nsafe + ib;
            const int past = nv + g.nsafe - v0;  // (no footprint goes further)
            if (past <= 0) continue;
            v0 += v0 < 0 ? nv : 0;
            v0 -= v0 >= nv ? nv : 0;
            const int first = wsg::band_col(v0, Lv, nv);
            for (int c = 0; c + ib < n && c < past; ++c) {
              const int got = wsg::band_col_next(first, c, nv, nvs), v = (v0 + c) % nv;
              int want = v;
              if (g.vprune) want = v <= Lv ? v + Lv : (nv - v <= Lv ? v - nv + Lv : -1);
              // (the row may have one entry of padding after column Lv)
              const bool pad = want < 0 && got == 2 * Lv + 1 && got < nvs;
              if (first < 0 || first >= 65536 || (got != want && !pad)) ++wrong;
            }
          }
      }
  std::printf("%ld %ld %ld %ld %ld\n", wrong, pruned, both, whole, small);
  return 0;
}
'''


def test_columns_of_every_tile(tmp_path):
    src = tmp_path / "columns.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "columns"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    str(src), os.path.join(CSRC, "es_kernel.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    wrong, pruned, both, whole, small = (int(x) for x in out.split())
    assert pruned > 50 and both > 20 and whole > 0 and small > 20, out
    assert wrong == 0, out
