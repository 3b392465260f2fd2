"""The tensor-core sweep's tail: the last unit of a CTA finished by four
epilogue warps, earlier ones by the finalizer warp, one split and several.
Tolerances are helpers.assert_parity's."""
import pytest

from tests import helpers, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,d", [
    (1, 1, 64), (129, 700, 40),     # a row block of one row; several splits
    (300, 9001, 64),                # splits of few row blocks; row blocks of few splits
    (30001, 257, 64),               # more row blocks than CTAs: one and two units a CTA
    (1025, 1100, 128),
])
def test_tail_of_the_sweep(n, m, d):
  x, y, a, b = problems.gaussian_shift_problem(n, m, d, seed=n)
  kw = dict(epsilon=0.5, relative_epsilon="mean", max_iterations=20)
  geom, out = helpers.gpu_solve(x, y, a, b, **kw)
  ref = helpers.oracle_solve(x, y, a, b, batch_size=1024, **kw)
  helpers.assert_parity(geom, out, ref)


def test_same_bits_again():
  """Which warps finish a row block may differ from run to run (units are
  drawn from a queue); the sums they take do not."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  ps = [problems.gaussian_shift_problem(900 + 57 * k, 1500 - 31 * k, 32, seed=k) for k in range(12)]
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geoms = [pointcloud.PointCloud(cu(p[0]), cu(p[1]), epsilon=20.0) for p in ps]
  runs = [linear.solve_batch(geoms, [cu(p[2]) for p in ps], [cu(p[3]) for p in ps],
                             max_iterations=30) for _ in range(3)]
  for k in range(len(ps)):
    for run in runs[1:]:
      assert torch.equal(run[k].f, runs[0][k].f) and torch.equal(run[k].g, runs[0][k].g)
      assert run[k].reg_ot_cost == runs[0][k].reg_ot_cost
      assert torch.equal(run[k].errors, runs[0][k].errors)
