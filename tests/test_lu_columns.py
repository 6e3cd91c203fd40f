"""csrc/kls_lu_cols.h run on the host.  The column schedule of the pipelined LU: over all
warps of a cluster every column is factored once, in order, and none that the matrix
does not have; the warp that keeps the determinant takes in all n of them.  And the rule
between it and one CTA per matrix, against measured times."""
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


# N, matrices, clusters in a wave, us a column and wave (lup_classes), us of the pipelined
# form, us of one CTA per matrix (B200, both forms' kernels alone)
MEASURED = [
    (41, 1, 71, 0.84, 37, 86), (41, 16, 71, 0.84, 38, 87),
    (41, 64, 71, 0.84, 39, 88), (41, 96, 71, 0.84, 72, 89),
    (41, 148, 71, 0.84, 103, 89), (41, 296, 71, 0.84, 169, 173),
    (41, 1184, 71, 0.84, 569, 668), (101, 1, 22, 1.08, 97, 296),
    (101, 16, 22, 1.08, 99, 298), (101, 64, 45, 1.08, 240, 299),
    (101, 96, 45, 1.08, 346, 299), (101, 148, 45, 1.08, 462, 302),
    (101, 296, 45, 1.08, 823, 595), (101, 1184, 45, 1.08, 3174, 2387),
    (128, 1, 22, 1.08, 134, 461), (128, 16, 22, 1.08, 136, 465),
    (128, 64, 45, 1.08, 300, 465), (128, 96, 45, 1.08, 438, 468),
    (128, 148, 45, 1.08, 590, 476), (128, 296, 45, 1.08, 1058, 939),
    (128, 1184, 45, 1.08, 4073, 3758), (150, 1, 22, 1.41, 205, 731),
    (150, 16, 22, 1.41, 208, 742), (150, 64, 22, 1.41, 618, 746),
    (150, 96, 22, 1.41, 1021, 748), (150, 148, 22, 1.41, 1430, 756),
    (150, 296, 22, 1.41, 2852, 1504), (150, 1184, 22, 1.41, 11012, 5903),
    (201, 1, 22, 1.71, 344, 1537), (201, 16, 22, 1.71, 348, 1570),
    (201, 64, 22, 1.71, 1029, 1588), (201, 96, 22, 1.71, 1703, 1621),
    (201, 148, 22, 1.71, 2389, 1969), (201, 296, 22, 1.71, 4764, 3684),
    (201, 1184, 22, 1.71, 18421, 13573), (256, 1, 15, 1.77, 449, 2680),
    (256, 16, 15, 1.77, 904, 2723), (256, 64, 15, 1.77, 2255, 2739),
    (256, 96, 15, 1.77, 3154, 3413), (256, 148, 15, 1.77, 4523, 4973),
    (256, 296, 15, 1.77, 9035, 9687), (256, 1184, 15, 1.77, 35688, 33856),
    (301, 1, 11, 1.8, 550, 4367), (301, 16, 11, 1.8, 1097, 4502),
    (301, 64, 11, 1.8, 3298, 4988), (301, 96, 11, 1.8, 4946, 6708),
    (301, 148, 11, 1.8, 7676, 9303), (301, 296, 11, 1.8, 14845, 18066),
    (301, 1184, 11, 1.8, 59219, 67556), (360, 1, 7, 2.9, 1077, 7061),
    (360, 16, 7, 2.9, 3187, 7243), (360, 64, 7, 2.9, 10622, 9847),
    (360, 96, 7, 2.9, 14903, 12261), (360, 148, 7, 2.9, 23360, 16550),
    (360, 296, 7, 2.9, 45711, 32491), (360, 1184, 7, 2.9, 180479, 124929),
    (400, 1, 7, 2.9, 1249, 9317), (400, 16, 7, 2.9, 3658, 9663),
    (400, 64, 7, 2.9, 12201, 14059), (400, 96, 7, 2.9, 17104, 16783),
    (400, 148, 7, 2.9, 26828, 22673), (400, 296, 7, 2.9, 52498, 44523),
    (400, 1184, 7, 2.9, 207233, 173511), (512, 1, 7, 4.0, 2937, 17966),
    (512, 16, 7, 4.0, 6513, 18239), (512, 64, 7, 4.0, 21676, 30392),
    (512, 96, 7, 4.0, 30441, 35600), (512, 148, 7, 4.0, 47724, 47366),
    (512, 296, 7, 4.0, 93312, 93671), (512, 1184, 7, 4.0, 368551, 368984),
]
RULE = r"""
#include "kls_lu_cols.h"
#include <cstdio>
int main() {
  int N, n, clusters;
  double us;
  while (scanf("%d %d %d %lf", &N, &n, &clusters, &us) == 4)
    printf("%d\n", (int)lup_wins(n, N, clusters, us, 148));
  return 0;
}
"""


def test_rule_takes_the_faster_form(tmp_path):
    """At most 15% behind the faster one anywhere; never the slower one for one matrix."""
    exe = tmp_path / "rule"
    (tmp_path / "rule.cpp").write_text(RULE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "kalnajs_log_spirals_b200", "csrc"),
                    str(tmp_path / "rule.cpp"), "-o", str(exe)], check=True)
    text = "".join("%d %d %d %g\n" % row[:4] for row in MEASURED)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True)
    for row, wins in zip(MEASURED, out.stdout.split()):
        N, n, _, _, pipe, cta = row
        chosen = pipe if wins == "1" else cta
        assert chosen <= 1.15 * min(pipe, cta), row
        assert n > 1 or wins == "1", row
