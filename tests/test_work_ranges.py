"""Contiguous ranges of work items (chunk < 0): every item once, ascending, ranges that differ by one item at most."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SOURCE = r"""
#include "work_walk.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** argv) {
  const int total = std::atoi(argv[1]), grid = std::atoi(argv[2]), stages = 3;
  int expect = 0;
  for (int cta = 0; cta < grid; ++cta) {
    gw::SegmentWalk walk(cta, grid, false, total, stages, -1);
    int tile, ks0, ks1, taken = 0;
    bool start;
    while (walk.next(tile, ks0, ks1, start)) {
      if (tile != expect++ || ks0 != 0 || ks1 != stages) return 1;
      ++taken;
    }
    if (taken < total / grid || taken > total / grid + 1) return 2;
  }
  return expect == total ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("total,grid", [(0, 1), (1, 148), (147, 148), (148, 148), (149, 148), (2816, 148), (65537, 7)])
def test_contiguous_ranges(tmp_path, total, grid):
    (tmp_path / "walk.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "gewell_b200" / "csrc"), str(tmp_path / "walk.cpp"), "-o", str(tmp_path / "walk")], check=True)
    assert subprocess.run([str(tmp_path / "walk"), str(total), str(grid)]).returncode == 0
