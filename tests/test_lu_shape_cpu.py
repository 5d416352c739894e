"""CPU: the LU panel's cluster keeps to the CTAs that the device can place (8 everywhere, 16 on a
whole B200), with enough rows and at most four per thread, for every number of rows."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include "lu_shape.h"
int main() {
  for (int top = 8; top <= 16; top *= 2)
    for (int m = 1; m <= mo::cl_max_rows(top); ++m) {
      int r = 0;
      const int c = mo::cl_shape(m, top, &r);
      const bool shape = c <= top && (r == 1 || r == 2 || r == mo::kClMaxRpt);
      // no more CTAs than the rows need, and a second row per thread only in the largest cluster
      if (!shape || (long)c * mo::kClThreads * r < m || (r > 1 && c != top) ||
          (c > 1 && (long)c / 2 * mo::kClThreads * r >= m && r == 1)) {
        std::printf("%d rows, at most %d CTAs: %d CTAs, %d rows per thread\n", m, top, c, r);
        return 1;
      }
    }
  return mo::cl_max_rows(8) == 8192 && mo::cl_max_rows(16) == 16384 ? 0 : 2;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_shapes(tmp_path):
    src = tmp_path / "shape.cpp"
    src.write_text(MAIN)
    exe = tmp_path / "shape"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "matops_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
