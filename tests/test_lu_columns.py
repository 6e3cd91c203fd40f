"""The column schedule of the pipelined LU (csrc/kls_lu_cols.h) run on the host: over all
warps of a cluster every column is factored once, in order, and none that the matrix
does not have; the warp that keeps the determinant takes in all n of them."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

MAIN = r"""
#include "kls_lu_cols.h"
#include <cstdio>
#include <cstdlib>
#include <vector>
int main(int, char** v) {
  const int n = atoi(v[1]), C = atoi(v[2]), LP = atoi(v[3]);
  std::vector<int> factored(n + 1, 0);
  for (int rank = 0; rank < C; ++rank)
    for (int warp = 0; warp < LUP_WARPS; ++warp) {
      const bool keeper = rank == 0 && warp == 0;
      LupCols own(n, C, rank, warp, LP);
      if (own.next == 0) { ++factored[0]; own.taken(); }
      for (int j = 0; j < (keeper ? n : own.last); ++j)
        if (own.next == j + 1) {                 // as lup_body's chain does
          ++factored[own.next];
          own.taken();
        }
      if (own.left != 0) { printf("rank %d warp %d: %d left\n", rank, warp, own.left); return 1; }
    }
  for (int g = 0; g <= n; ++g)
    if (factored[g] != (g < n)) { printf("column %d factored %d times\n", g, factored[g]); return 1; }
  return 0;
}
"""


@pytest.mark.parametrize("n,C,LP", [(1, 4, 2), (8, 4, 2), (9, 4, 2), (33, 4, 2), (64, 4, 2),
                                    (101, 6, 3), (128, 6, 3), (192, 12, 2), (201, 6, 5),
                                    (256, 16, 2), (301, 10, 4), (320, 10, 4), (512, 16, 4)])
def test_every_column_is_factored_once(tmp_path, n, C, LP):
    exe = tmp_path / "cols"
    (tmp_path / "cols.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "kalnajs_log_spirals_b200", "csrc"),
                    str(tmp_path / "cols.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(n), str(C), str(LP)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
