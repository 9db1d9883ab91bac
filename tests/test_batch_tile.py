"""The batch's cut of a site's slices into tiles, on the CPU: with right-hand sides one after the other a tile
holds whole ones or a whole part of one, and every such cut that the split allows is taken."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROG = r"""
#include "batch_tile.h"
#include <cstdio>
int main() {
  for (int Ls = 1; Ls <= 24; ++Ls)
    for (int nrhs = 1; nrhs <= 12; ++nrhs)
      for (int spt = 1; spt <= 2; ++spt)
        for (int split = 1; split <= 32; split *= 2)
          if (Ls * nrhs % spt == 0) std::printf("%d %d %d %d %d\n", Ls, nrhs, spt, split, gbdw::batch_tile(Ls * nrhs, Ls, spt, split));
}
"""


def test_tiles_hold_whole_right_hand_sides_or_parts_of_one(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROG)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "gridbench_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    seen = {}
    for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines():
        Ls, nrhs, spt, split, te = map(int, line.split())
        fits = [Ls * nrhs // sp for sp in (32, 16, 8, 4, 2) if sp <= split and Ls * nrhs % sp == 0]
        fits = [t for t in fits if t % spt == 0 and (t % Ls == 0 or Ls % t == 0)]
        assert te == (fits[0] if fits else Ls * nrhs), line
        seen[Ls, nrhs, spt, split] = te
    assert seen[12, 8, 2, 8] == 12  # one right-hand side each
    assert seen[12, 8, 2, 16] == 6
    assert seen[8, 6, 2, 16] == 24  # 6 and 12 slices would straddle two
