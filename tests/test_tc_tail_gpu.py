"""The tensor-core sweep's tail: the last unit of a CTA finished by four
epilogue warps, earlier ones by the finalizer warp, one split and several.
Tolerances are helpers.assert_parity's."""
import pytest

from tests import helpers, problems

@pytest.mark.gpu
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


@pytest.mark.gpu
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


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,d", [
    (10007, 7919, 50),    # f: runs of 16 and 17 tiles, up to 3 CTAs in a row block; g: 2 splits
    (20011, 5003, 33),    # g: runs that end inside row blocks of one row
    (38000, 1100, 128),   # runs longer than a row block
])
def test_runs_of_tiles(n, m, d):
  x, y, a, b = problems.gaussian_shift_problem(n, m, d, seed=n)
  kw = dict(epsilon=0.5, relative_epsilon="mean", max_iterations=10)
  geom, out = helpers.gpu_solve(x, y, a, b, **kw)
  ref = helpers.oracle_solve(x, y, a, b, batch_size=1024, **kw)
  helpers.assert_parity(geom, out, ref)


@pytest.mark.parametrize("grid", [7, 148])
def test_runs_cover_every_tile_once(grid):
  """The dealer's arithmetic (host restatement): units of consecutive runs
  tile every row block, S counts them and sidx numbers them."""
  for rb, nt in ((79, 31), (40, 157), (297, 5), (512, 256), (149, 20), (5, 149), (600, 1)):
    tiles = rb * nt
    if tiles // grid < 4:
      continue
    met = {}
    for c in range(grid):
      pos, end = tiles * c // grid, tiles * (c + 1) // grid
      while pos < end:
        r = pos // nt
        stop = (r + 1) * nt
        first = ((stop - nt + 1) * grid - 1) // tiles
        last = (stop * grid - 1) // tiles
        met.setdefault(r, []).append((c - first, last - first + 1, pos - (stop - nt),
                                      min(stop, end) - (stop - nt)))
        pos = min(stop, end)
    assert sorted(met) == list(range(rb))
    run = tiles // grid
    for units in met.values():
      assert [u[0] for u in units] == list(range(len(units)))
      assert all(u[1] == len(units) for u in units)
      assert len(units) <= (nt + run - 2) // run + 1 <= max(nt, 1)
      assert units[0][2] == 0 and units[-1][3] == nt
      assert all(p[3] == q[2] for p, q in zip(units, units[1:]))
