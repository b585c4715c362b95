"""The convolution's row ring counts a row only once its wait has succeeded, so that
after a wait that ran out the drain starts at the row still in flight (compiled for the
host: no such wait is provoked on a GPU)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "seistorch_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "row_ring.cuh"
int main() {
  for (int fail = 0; fail < 12; ++fail) {  // the row whose wait runs out
    int rows = 0, asked = 0;
    bool ok = true;
    for (int tile = 0; tile < 8 && ok; ++tile)
      ok = sgb::nn::take_rows(tile == 0 || tile == 4 ? 3 : 1, rows, [&](int row) { asked = row; return row != fail; });
    printf("%d %d %d %d\n", fail, (int)ok, rows, asked);
  }
}
"""


def test_a_row_that_did_not_arrive_is_not_counted(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs a host compiler")
    (tmp_path / "ring.cpp").write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", f"-I{CSRC}", "-o", tmp_path / "ring", tmp_path / "ring.cpp"], check=True)
    out = subprocess.run([tmp_path / "ring"], check=True, capture_output=True, text=True).stdout
    for line in out.splitlines():
        fail, ok, rows, asked = map(int, line.split())
        assert (ok, rows, asked) == (0, fail, fail)  # 12 rows in all: every `fail` is met
