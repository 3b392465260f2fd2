"""The FP32 row-owner engine against the float64 oracle where its split of
the work changes: single CTAs, clusters and the whole grid, columns resident
and streamed, several passes over the columns, remainders of quads and
tiles, every padded dimension, potentials exchanged by words and behind the
barrier. Tolerances are the FP32 path's (helpers.assert_parity)."""
import numpy as np
import pytest

from tests import helpers, problems

pytestmark = pytest.mark.gpu


def _check(n, m, d, seed, **kw):
  x, y, a, b = problems.uniform_cloud_problem(n, m, d, seed=seed)
  geo = dict(epsilon=0.05, relative_epsilon="mean")
  geom, out = helpers.gpu_solve(x, y, a, b, precision="fp32", **geo, **kw)
  ref = helpers.oracle_solve(x, y, a, b, batch_size=1024, **geo, **kw)
  helpers.assert_parity(geom, out, ref)


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16])
@pytest.mark.parametrize("n,m", [(45, 70), (1501, 1303)])
def test_dimensions(n, m, d):
  """One CTA or a small cluster; the grid with resident columns."""
  _check(n, m, d, seed=d)


@pytest.mark.parametrize("n,m,d", [
    (1, 1, 2), (1, 300, 3), (300, 1, 3), (3, 5, 4), (129, 33, 2),   # fewer rows than CTAs
    (511, 513, 2), (900, 1100, 2),                                  # clusters
    (2900, 3101, 3), (3007, 2999, 16),        # grid: words; streamed columns
    (5001, 4003, 2), (2049, 8193, 5),         # grid: the barrier, resident; streamed, a short chunk
    (60013, 37, 2), (29, 58001, 3),           # several passes; skewed sizes
])
def test_sizes(n, m, d):
  _check(n, m, d, seed=n)


@pytest.mark.parametrize("n,m,d", [(60, 45, 3), (700, 400, 2), (2500, 2600, 3), (6001, 5003, 2)])
def test_epsilon_decay_and_late_blocks(n, m, d):
  """Multipliers other than 1 (the exchange of potentials instead of
  shifts), blocks whose error is not asked for, a marginal sweep of its own
  at the end."""
  import torch
  from oracle import sinkhorn_np as oracle
  from ott_b200.geometry import epsilon_scheduler, pointcloud
  from ott_b200.solvers import linear
  x, y, a, b = problems.uniform_cloud_problem(n, m, d, seed=5)
  for kw in (dict(), dict(min_iterations=25), dict(max_iterations=15, inner_iterations=5,
                                                   min_iterations=15)):
    eps = epsilon_scheduler.Epsilon(target=0.02, init=20.0, decay=0.7)
    geom = pointcloud.PointCloud(torch.as_tensor(x).cuda(), torch.as_tensor(y).cuda(), epsilon=eps)
    out = linear.solve(geom, torch.as_tensor(a).cuda(), torch.as_tensor(b).cuda(), **kw)
    ref = oracle.solve(x, y, a, b, epsilon=0.02, eps_init=20.0, eps_decay=0.7, batch_size=1024,
                       **kw)
    assert out.n_iters == ref.n_iters
    helpers.assert_parity(geom, out, ref)


def test_batch_of_every_team():
  """One call whose problems go to clusters and, the large ones, to the
  grid; the clusters solve several problems one after another."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  sizes = [(7, 9), (40, 300), (3000, 2500), (129, 128), (1, 4), (600, 601), (64, 5000)] + \
      [(90 + 7 * k, 210 - 3 * k) for k in range(40)]
  ps = [problems.uniform_cloud_problem(n, m, 3, seed=i) for i, (n, m) in enumerate(sizes)]
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geoms = [pointcloud.PointCloud(cu(p[0]), cu(p[1]), epsilon=0.02) for p in ps]
  outs = linear.solve_batch(geoms, [cu(p[2]) for p in ps], [cu(p[3]) for p in ps])
  for p, geom, out in zip(ps, geoms, outs):
    ref = helpers.oracle_solve(*p, epsilon=0.02, batch_size=1024)
    helpers.assert_parity(geom, out, ref)


def test_zero_weights_of_a_whole_quad():
  """Rows and columns at -inf, a quad of them at a time."""
  x, y, a, b = problems.uniform_cloud_problem(1300, 1500, 3, seed=2)
  a[8:12] = 0
  b[:5] = 0
  b[-3:] = 0
  a, b = (a / a.sum()).astype(np.float32), (b / b.sum()).astype(np.float32)
  kw = dict(epsilon=0.05, relative_epsilon="mean")
  geom, out = helpers.gpu_solve(x, y, a, b, **kw)
  ref = helpers.oracle_solve(x, y, a, b, **kw)
  helpers.assert_parity(geom, out, ref)


@pytest.mark.parametrize("n,m,d", [
    (2900, 3101, 10), (4099, 2050, 9), (4801, 4700, 10),  # near the buffer's limits
    (2901, 2803, 16), (3503, 2600, 12),
    (6007, 301, 8), (37, 6201, 8),                        # skewed: few rows, or CTAs without any
])
def test_columns_in_turns(n, m, d):
  """Both sides' points do not fit in shared memory together, either does."""
  _check(n, m, d, seed=m)


@pytest.mark.parametrize("kw", [dict(), dict(min_iterations=25),
                                dict(max_iterations=15, inner_iterations=5, min_iterations=15)])
def test_columns_in_turns_order_of_sweeps(kw):
  """Multipliers other than 1 and blocks that evaluate without an update."""
  import torch
  from oracle import sinkhorn_np as oracle
  from ott_b200.geometry import epsilon_scheduler, pointcloud
  from ott_b200.solvers import linear
  x, y, a, b = problems.uniform_cloud_problem(3100, 3302, 9, seed=5)
  eps = epsilon_scheduler.Epsilon(target=0.05, init=10.0, decay=0.7)
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geom = pointcloud.PointCloud(cu(x), cu(y), epsilon=eps)
  out = linear.solve(geom, cu(a), cu(b), **kw)
  ref = oracle.solve(x, y, a, b, epsilon=0.05, eps_init=10.0, eps_decay=0.7, batch_size=1024, **kw)
  assert out.n_iters == ref.n_iters
  helpers.assert_parity(geom, out, ref)


def test_columns_in_turns_batch():
  """Several problems of one call through the same buffer."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  kw = dict(max_iterations=10)
  ps = [problems.uniform_cloud_problem(n, m, 4, seed=n) for n, m in [(4901, 4902), (4850, 5003)]]
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geoms = [pointcloud.PointCloud(cu(p[0]), cu(p[1]), epsilon=0.05) for p in ps]
  outs = linear.solve_batch(geoms, [cu(p[2]) for p in ps], [cu(p[3]) for p in ps], **kw)
  for p, geom, out in zip(ps, geoms, outs):
    ref = helpers.oracle_solve(*p, epsilon=0.05, batch_size=1024, **kw)
    helpers.assert_parity(geom, out, ref)


@pytest.mark.parametrize("inner", [1, 10])
@pytest.mark.parametrize("n,m", [(4000, 200), (200, 4000), (1000, 40), (4000, 8), (8, 4000), (9, 5)])
def test_team_members_without_rows(n, m, inner):
  """CTAs of a grid or cluster that own rows of one side only, or of none:
  they take no part in the other side's exchange and meet the others in the
  evaluating sweeps."""
  _check(n, m, 2, seed=n + m, inner_iterations=inner)


def test_batch_with_members_without_rows():
  """Clusters that draw problems with fewer quads of rows than CTAs between
  larger ones."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  sizes = [(1500, 1400), (1300, 9), (7, 1200), (5, 6), (900, 30), (1, 1), (1100, 1000)]
  ps = [problems.uniform_cloud_problem(n, m, 3, seed=i) for i, (n, m) in enumerate(sizes)]
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geoms = [pointcloud.PointCloud(cu(p[0]), cu(p[1]), epsilon=0.05) for p in ps]
  outs = linear.solve_batch(geoms, [cu(p[2]) for p in ps], [cu(p[3]) for p in ps])
  for p, geom, out in zip(ps, geoms, outs):
    helpers.assert_parity(geom, out, helpers.oracle_solve(*p, epsilon=0.05, batch_size=1024))


@pytest.mark.parametrize("inner,its", [(1, 7), (3, 12)])
def test_streamed_bound_across_evaluating_sweeps(inner, its):
  """The streamed sweeps' bound on the change of the column shifts, with an
  evaluating sweep before every update and before some."""
  _check(6001, 5003, 10, seed=3, inner_iterations=inner, max_iterations=its)


def _check_symmetric(n, d, eps, **kw):
  """The parallel, momentum-1/2 update on x = y, a = b."""
  import torch
  from oracle import sinkhorn_np as oracle
  from ott_b200.geometry import pointcloud
  from ott_b200.problems.linear import linear_problem
  from ott_b200.solvers.linear import acceleration, sinkhorn
  x, _, a, _ = problems.uniform_cloud_problem(n, n, d, seed=n)
  xt, at = torch.as_tensor(x).cuda(), torch.as_tensor(a).cuda()
  geom = pointcloud.PointCloud(xt, xt, epsilon=eps)
  solver = sinkhorn.Sinkhorn(parallel_dual_updates=True, precision="fp32",
                             momentum=acceleration.Momentum(start=0, value=0.5), **kw)
  x64, a64 = x.astype(np.float64), a.astype(np.float64)
  out = solver(linear_problem.LinearProblem(geom, at, at))
  ref = helpers.oracle_sinkhorn(oracle.Geom(x64, x64, eps, batch_size=1024), a64, a64,
                                parallel_dual_updates=True, momentum=0.5, **kw)
  helpers.assert_parity(geom, out, ref)


@pytest.mark.parametrize("n", [30, 700, 2501, 5002])
def test_symmetric_blocks_of_one_iteration(n):
  """Every sweep evaluates; nothing is exchanged between two sums but the
  sums themselves."""
  _check_symmetric(n, 2, 0.05, inner_iterations=1, max_iterations=15)


@pytest.mark.parametrize("n,d,eps", [(1102, 2, 0.004), (2303, 3, 0.003), (5901, 10, 0.02)])
def test_symmetric_from_given_potentials(n, d, eps):
  """A warm start from 100 times the epsilon, whose first updates move the
  column shifts by hundreds of log2 units: clusters, the grid's resident and
  streamed columns. Ten iterations leave an error at the level of the FP32
  exponents' rounding (the largest |f - |x|^2| / eps is 150 to 600, times
  2^-24: 1e-5 to 4e-5 of a row's mass), so what is compared is the potentials,
  within the FP32 path's 1e-4 eps."""
  import torch
  from oracle import sinkhorn_np as oracle
  from ott_b200.geometry import pointcloud
  from ott_b200.problems.linear import linear_problem
  from ott_b200.solvers.linear import acceleration, sinkhorn
  x, _, a, _ = problems.uniform_cloud_problem(n, n, d, seed=n)
  x64, a64 = x.astype(np.float64), a.astype(np.float64)
  kw = dict(min_iterations=10, max_iterations=10, parallel_dual_updates=True)
  warm = oracle.sinkhorn(oracle.Geom(x64, x64, 100 * eps, batch_size=1024), a64, a64,
                         momentum=0.5, **kw).f.astype(np.float32)
  xt, at, wt = (torch.as_tensor(t).cuda() for t in (x, a, warm))
  solver = sinkhorn.Sinkhorn(momentum=acceleration.Momentum(start=0, value=0.5),
                             precision="fp32", **kw)
  geom = pointcloud.PointCloud(xt, xt, epsilon=eps)
  out = solver(linear_problem.LinearProblem(geom, at, at), init=(wt, wt))
  ref = oracle.sinkhorn(oracle.Geom(x64, x64, eps, batch_size=1024), a64, a64, momentum=0.5,
                        init=(warm, warm), **kw)
  helpers.assert_potentials(out.f.cpu().numpy().astype(np.float64),
                            out.g.cpu().numpy().astype(np.float64), ref, 1e-4)


@pytest.mark.parametrize("n,m,d", [(1000, 1100, 2), (2048, 2000, 3), (2050, 2040, 5), (30001, 700, 3)])
def test_side_without_weight(n, m, d):
  """Every column of the other side's sweeps at -inf: a row's log-sum-exp is
  -inf under the running maximum and under the bounded shift, with part of
  the exponentials on the polynomial (d <= 3) and without."""
  x, y, _, b = problems.uniform_cloud_problem(n, m, d, seed=2)
  kw = dict(epsilon=0.05, max_iterations=20)
  _, out = helpers.gpu_solve(x, y, np.zeros(n, np.float32), b, precision="fp32", **kw)
  ref = helpers.oracle_solve(x, y, np.zeros(n), b, batch_size=1024, **kw)
  helpers.assert_potentials(out.f.cpu().numpy().astype(np.float64),
                            out.g.cpu().numpy().astype(np.float64), ref, 1e-4)
  # every marginal is 0: the error is the other side's mass
  np.testing.assert_allclose(out.errors.cpu().numpy(), ref.errors, rtol=1e-5)


def _sinkhorn64(x, y, a, b, eps, iterations):
  """The float64 iteration in plain torch, for sizes that take numpy minutes:
  potentials and the last error (of the g marginal)."""
  import torch

  def lse(p, q, pot):  # eps log sum_j exp((pot_j - C_ij) / eps), rows of p
    out = torch.empty(p.shape[0], dtype=torch.float64, device=p.device)
    for i in range(0, p.shape[0], 1024):
      c = (p[i:i + 1024] ** 2).sum(1, keepdim=True) + (q ** 2).sum(1) - 2.0 * p[i:i + 1024] @ q.T
      out[i:i + 1024] = eps * torch.logsumexp((pot - c) / eps, dim=1)
    return out

  x, y, a, b = (torch.as_tensor(t).cuda().double() for t in (x, y, a, b))
  f, g = torch.zeros_like(a), torch.zeros_like(b)
  for _ in range(iterations):
    g = eps * b.log() - lse(y, x, f)
    f = eps * a.log() - lse(x, y, g)
  err = (torch.exp((lse(y, x, f) + g) / eps) - b).abs().sum()
  return f, g, float(err)


@pytest.mark.parametrize("n,m,d", [
    (30000, 30000, 10), (65536, 65536, 8), (500, 40000, 10), (51700, 51600, 7),  # own rows not kept
    (700001, 100, 9), (950001, 100, 10), (2001, 600001, 10),                     # shorter passes
])
def test_large_streamed_dimensions(n, m, d):
  """Two chunks of d = 7 ... 10 leave little of a CTA's shared memory for
  the rest of its layout."""
  x, y, a, b = problems.uniform_cloud_problem(n, m, d, seed=n + d)
  eps, its = 0.05, 3
  _, out = helpers.gpu_solve(x, y, a, b, precision="fp32", epsilon=eps, min_iterations=its,
                             max_iterations=its, inner_iterations=its)
  f, g, err = _sinkhorn64(x, y, a, b, eps, its)
  np.testing.assert_allclose(out.f.cpu().numpy(), f.cpu().numpy(), rtol=0, atol=1e-4 * eps)
  np.testing.assert_allclose(out.g.cpu().numpy(), g.cpu().numpy(), rtol=0, atol=1e-4 * eps)
  np.testing.assert_allclose(float(out.errors[0]), err, rtol=1e-2, atol=1e-6)


@pytest.mark.parametrize("d", [1, 2, 3, 4])
@pytest.mark.parametrize("n,m", [(150, 40001), (60003, 200)])
def test_short_sides_of_long_problems(n, m, d):
  """Left to the tiled engine, at its smallest dimensions."""
  _check(n, m, d, seed=d, max_iterations=20)


def test_batch_of_long_problems():
  """Several problems that would take the whole grid one after another: the
  tiled engine, with small ones between."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  ps = [problems.uniform_cloud_problem(n, m, 3, seed=n)
        for n, m in [(20000, 30), (20003, 301), (45, 21000), (300, 200)]]
  cu = lambda t: torch.as_tensor(t).cuda()  # noqa: E731
  geoms = [pointcloud.PointCloud(cu(p[0]), cu(p[1]), epsilon=0.05) for p in ps]
  outs = linear.solve_batch(geoms, [cu(p[2]) for p in ps], [cu(p[3]) for p in ps])
  for p, geom, out in zip(ps, geoms, outs):
    helpers.assert_parity(geom, out, helpers.oracle_solve(*p, epsilon=0.05, batch_size=1024))
