"""Which cells the non-reflecting edges' offsets reach (csrc/bc_offset.h), on the
host: the classification against every sector's target, for offsets around each
whole number of turns, the largest that fit, infinities and NaN."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cudaprotoplanetarydisksfloat_b200", "csrc")

SRC = r'''
#include <cmath>
#include <cstdio>
#include "bc_offset.h"
int main() {
  long bad = 0, seen[4] = {0, 0, 0, 0};
  const int grids[][2] = {{4, 129}, {5, 130}, {8, 131}, {12, 260}};
  for (auto& g : grids) {
    const int nrad = g[0], n = g[1];
    const long long cells = (nrad + 1LL) * n;
    for (int t = -nrad - 3; t <= nrad + 3; t++)
      for (int s = -2; s <= 2; s++)
        for (int t2 = -nrad - 3; t2 <= nrad + 3; t2++)
          for (int s2 = -2; s2 <= 2; s2++) {
            const int a = t * n + s, a2 = t2 * n + s2;
            bool ring = true, rows = true;
            for (int j = 0; j < n; j++) {
              const long long w = bc_wrap(j, a, n), r = bc_wrap(j, -a2, n);
              ring &= w >= 0 && w < n && r >= 0 && r < n;
              const long long c = (nrad - 2LL) * n + r;
              rows &= w >= 0 && w < cells && c >= 0 && c < cells;
            }
            const BcReach want = ring ? kBcInRing : rows ? kBcInRows : kBcOutside;
            // the fraction is dropped toward zero, as the conversion does
            const double f = a < 0 ? -0.5 : 0.5, f2 = a2 < 0 ? -0.25 : 0.25;
            const BcReach got = bc_reach(a + f, a2 + f2, nrad, n);
            bad += got != want;
            seen[got]++;
          }
  }
  const double big[] = {INFINITY, -INFINITY, 1e300, -1e300, 2147483647.0, -2147483648.0, 4.3e9};
  for (double x : big) bad += bc_reach(x, 0, 16, 130) != kBcOutside, bad += bc_reach(0, x, 16, 130) != kBcOutside;
  bad += bc_reach(NAN, 0, 16, 130) != kBcNotFinite;
  bad += bc_reach(INFINITY, NAN, 16, 130) != kBcNotFinite;
  std::printf("%ld %ld %ld %ld\n", bad, seen[kBcInRing], seen[kBcInRows], seen[kBcOutside]);
}
'''


def test_reach_against_every_target(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I" + CSRC, str(src), "-o", str(exe)])
    bad, ring, rows, outside = map(int, subprocess.check_output([str(exe)]).split())
    assert bad == 0
    assert ring and rows and outside
