"""The row-owner engine's shared-memory layout: a streamed problem fits a
CTA at every size, dimension and team, so that no call is refused for it."""
import os
import subprocess

import pytest

from ott_b200 import build

_SRC = r"""
#include <cstdio>
#include "rows.h"
using namespace ottb;
int main() {
  const size_t limit = 224 * 1024;
  const int dims[] = {2, 3, 4, 5, 6, 8, 10, 12, 16};
  const int teams[] = {1, 2, 3, 7, 37, 64, 132, 147, 148};
  int bad = 0;
  for (int D : dims)
    for (int size : teams)
      for (double s = 1; s <= 1e6; s *= 1.05)
        for (double t = 1; t <= 1e6; t *= 1.31)
          for (int swap = 0; swap < 2; ++swap) {
            const int64_t n = (int64_t)(swap ? t : s), m = (int64_t)(swap ? s : t);
            // a team has no more CTAs than quads of rows
            if (size > 1 && size > ((n > m ? n : m) + 3) / 4) continue;
            const size_t b = rows_smem(n, m, D, size, kRowsWarps, false, false);
            const RowsLayout L = rows_layout(n, m, D, size, kRowsWarps, false, false, false);
            if (b > limit || L.rp < 1 || L.rp % 4) {
              if (bad++ < 10)
                printf("D %d, %d CTAs, n %lld, m %lld: %zu bytes, %d rows a pass\n", D, size,
                       (long long)n, (long long)m, b, L.rp);
            }
          }
  printf("%d\n", bad);
  return bad != 0;
}
"""


def test_streamed_layout_fits(tmp_path):
  try:
    nvcc = build.nvcc()
  except RuntimeError:
    pytest.skip("no nvcc")
  src, exe = tmp_path / "layout.cu", tmp_path / "layout"
  src.write_text(_SRC)
  subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I", build.CSRC, "-o", str(exe), str(src)],
                 check=True, capture_output=True, text=True)
  run = subprocess.run([str(exe)], capture_output=True, text=True, check=False,
                       env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
  assert run.returncode == 0, run.stdout
