"""Which engine an FP32 call takes, against sizes at which one of the two
measured clearly faster (B200; microseconds an iteration, tiled and
row-owner)."""
import os
import subprocess

import pytest

from ott_b200 import build

# n, m, number of problems, d, microseconds by the tiled and the row-owner engine
_MEASURED = [
    (200, 100000, 1, 2, 102, 182), (200, 100000, 1, 8, 138, 235), (100000, 200, 1, 4, 116, 205),
    (1200, 100000, 1, 8, 261, 360), (2400, 100000, 1, 8, 420, 546), (600, 100000, 1, 8, 211, 271),
    (300, 1000000, 1, 2, 1123, 1573), (150, 200000, 1, 3, 255, 363), (150, 200000, 1, 10, 389, 519),
    (130, 40000, 1, 4, 76, 90), (400, 200000, 1, 10, 485, 527), (1800, 1000000, 1, 8, 3120, 3702), (900, 200000, 1, 8, 447, 551),
    (20000, 30, 16, 2, 168, 679), (20000, 300, 16, 4, 261, 741), (20000, 1000, 16, 2, 398, 713),
    (100000, 8, 8, 2, 559, 1343), (100000, 500, 4, 2, 583, 672), (6000, 6000, 32, 2, 1106, 1305),
    (8, 4000, 1, 2, 64, 17), (4000, 200, 1, 2, 33, 20), (64, 100000, 1, 2, 1069, 177),
    (10, 100000, 1, 8, 1678, 226), (8, 1000000, 1, 4, 12891, 1853), (16000, 16000, 1, 4, 332, 250),
    (16000, 16000, 1, 8, 409, 357), (30000, 30000, 1, 10, 1839, 1178), (65536, 65536, 1, 8, 5902, 5250),
    (131072, 131072, 1, 10, 33565, 21469), (2000, 40000, 1, 3, 235, 117), (700, 10000, 1, 8, 48, 43),
    (9000, 40000, 1, 10, 873, 514), (12000, 200000, 1, 8, 3433, 2950), (20, 20000, 1, 2, 232, 47),
    (2048, 2048, 1, 2, 24, 14), (7013, 5001, 1, 3, 120, 60), (120, 96, 1, 3, 15, 7),
    (4000, 100, 64, 2, 135, 78), (8000, 8000, 4, 2, 301, 240), (60000, 1000, 2, 2, 341, 242),
    (300000, 300, 2, 4, 1575, 1094), (1024, 1024, 256, 2, 500, 320), (5000, 700, 64, 4, 383, 308),
]

_MAIN = r"""
#include <cstdio>
#include <vector>
#include "fp32_route.h"
using namespace ottb;
int main() {
  for (const auto& c : kMeasured) {
    std::vector<ottb_problem> p((size_t)c[2]);
    for (auto& q : p) q.n = c[0], q.m = c[1];
    const int d = (int)c[3];
    const int dims[] = {2, 3, 4, 5, 6, 8, 10, 12, 16};
    int D = 0, dp = 2;
    for (int k : dims)
      if (D == 0 && d <= k) D = k;
    while (dp < d) dp <<= 1;
    if (rows_wanted(p.data(), (int)p.size(), D, dp) != (c[5] < c[4]))
      printf("%lld x %lld, %lld problems, d %d\n", c[0], c[1], c[2], d);
  }
  // beyond 32-bit row numbers
  for (int64_t n : {((int64_t)1 << 30) + 1, (int64_t)1 << 31}) {
    ottb_problem q{};
    q.n = n, q.m = 10;
    if (rows_wanted(&q, 1, 2, 2)) printf("n %lld\n", (long long)n);
  }
}
"""


_TEAMS = r"""
#include <cstdio>
#include <vector>
#include "fp32_route.h"
using namespace ottb;
int main() {
  // a device that holds clusters of at most `fit` CTAs at once, or none
  for (int fit : {16, 8, 4, 2, 1, 0}) {
    auto clusters = [&](int size, int, size_t) { return size <= fit ? 9 : 0; };
    for (int num : {1, 3, 40}) {
      std::vector<RowsSize> p;
      for (int i = 0; i < num; ++i) p.push_back(RowsSize{1500 - 10 * i, 900, 148});
      const RowsTeams T = rows_teams(p, 3, 148, 2500, clusters);
      const bool on_grid = T.grid == num;
      if (on_grid ? T.nclusters != 0 : T.csize > fit || T.nclusters < 1 || !rows_fits(T.csmem))
        printf("fit %d, %d problems: grid %d, %d clusters of %d\n", fit, num, T.grid, T.nclusters,
               T.csize);
    }
  }
}
"""


def _run(tmp_path, source):
  try:
    nvcc = build.nvcc()
  except RuntimeError:
    pytest.skip("no nvcc")
  src, exe = tmp_path / "route.cu", tmp_path / "route"
  src.write_text(source)
  subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I", build.CSRC, "-o", str(exe), str(src)],
                 check=True, capture_output=True, text=True)
  run = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120,
                       env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
  assert run.stdout == "", run.stdout


def test_a_device_without_room_for_the_best_cluster(tmp_path):
  """Smaller clusters, or the grid: no call is refused for it."""
  _run(tmp_path, _TEAMS)


def test_route_takes_the_faster_engine(tmp_path):
  rows = ",".join("{%s}" % ",".join(map(str, c)) for c in _MEASURED)
  _run(tmp_path, "static const long long kMeasured[][6] = {%s};\n%s" % (rows, _MAIN))


_SMALL = r"""
#include <cstdio>
#include <vector>
#include "fp32_route.h"
using namespace ottb;
int main() {
  auto any = [](int, int, size_t) { return 64; };
  // a few problems: each has a cluster at once, faster than the grid in turn
  for (auto [n, m, num] : {std::tuple{2600, 2593, 4}, {2500, 2500, 5}, {3000, 2993, 6}, {3000, 2993, 8},
                           {3400, 3393, 6}, {2200, 2193, 4}}) {
    const RowsTeams T = rows_teams(std::vector<RowsSize>(num, {n, m, 148}), 2, 148, 2500, any);
    if (T.grid) printf("%d of %d x %d: %d on the grid\n", num, n, m, T.grid);
  }
  // many above d = 4: clusters of 16 leave too much to their ends
  for (auto [n, m] : {std::tuple{2500, 1000}, {1900, 1500}}) {
    const RowsTeams T = rows_teams(std::vector<RowsSize>(64, {n, m, 148}), 8, 148, 2500, any);
    if (T.grid || T.csize >= 16) printf("64 of %d x %d: grid %d, clusters of %d\n", n, m, T.grid, T.csize);
  }
}
"""


def test_teams_of_batches(tmp_path):
  """Batches that measured slower than by the tiled engine with other teams
  (iterations of 4 problems of 2600 x 2593, d = 2: 77 us tiled, 112 by the
  grid in turn, 47 in clusters; 64 of 2500 x 1000, d = 8: 313 tiled, 360 in
  clusters of 16, 229)."""
  _run(tmp_path, "#include <tuple>\n" + _SMALL)
