"""The work that this framework is measured on.

Each case is one call (or one training-style step) as a program makes it:
device arrays in hand, then the geometry, the solver and what the program
reads of the result. Sizes and distributions are those of the tests and of
``bench.py`` (uniform clouds, Gaussian clouds with a shift, Gaussian
mixtures, measures on a 32 x 32 grid) and generic ones between them.

Kinds of case:
  solve       ``linear.solve`` on one pair of clouds, from the geometry
              (epsilon relative to the mean or the spread of the cost) to the
              potentials, the error log, the cost and the iteration count
  batch       ``linear.solve_batch``: many pairs of uneven sizes, one launch
  stack       ``sinkhorn.run_stacked``: many weight pairs on one support
  divergence  ``sinkhorn_divergence`` and its gradient in the points
  implicit    a loss of the potentials and its gradient through the solve
  apply       the plan of given potentials applied to vectors
``iterations`` 0 solves to the default threshold; a positive number runs
that many iterations (``min_iterations == max_iterations``, the form whose
cost is known beforehand). ``about`` is the count that a solve to the
threshold takes, for ``work`` alone.
"""
import math
import random

import numpy as np
import torch

from ott_b200.geometry import epsilon_scheduler, pointcloud
from ott_b200.solvers import linear
from ott_b200.solvers.linear import sinkhorn
from ott_b200.tools import sinkhorn_divergence as sd

INNER = 10
THRESHOLD = 1e-3
MAX_ITERATIONS = 2000


def listed():
  solve = dict(kind="solve", relative="mean", scale_cost="", decay=1.0, precision="auto",
               iterations=0)
  return [
      # the smallest calls: a handful of points, every default of the
      # geometry (epsilon 0.05 std of the cost); latency and launches
      dict(solve, name="solve_120x96_d3", cloud="uniform", n=120, m=96, d=3, epsilon=0.0,
           relative="", about=100),
      # the reference's CPU-runnable configuration
      dict(solve, name="solve_2048_d2", cloud="uniform", n=2048, m=2048, d=2, epsilon=0.05,
           about=50),
      # two scans in space, ragged sizes
      dict(solve, name="solve_7013x5001_d3", cloud="uniform", n=7013, m=5001, d=3,
           epsilon=0.01, about=200),
      # tabular features, the cost scaled by its mean, epsilon in that unit
      dict(solve, name="solve_3000x4100_d10", cloud="gauss", n=3000, m=4100, d=10,
           epsilon=0.05, relative="", scale_cost="mean", about=50),
      # embeddings: an ordinary size, ragged sizes with an odd dimension, and
      # the headline size
      dict(solve, name="solve_4096_d64", cloud="gauss", n=4096, m=4096, d=64, epsilon=0.01,
           about=50),
      dict(solve, name="solve_10007x7919_d50", cloud="gauss", n=10007, m=7919, d=50,
           epsilon=0.02, about=30),
      dict(solve, name="solve_65536_d64", cloud="gauss", n=65536, m=65536, d=64, epsilon=0.01,
           about=30),
      # uneven pairs solved together
      dict(name="batch_96_d32", kind="batch", num=96, lo=128, hi=4096, d=32, epsilon=13.0,
           precision="auto", iterations=0, about=25),
      # weight pairs on one grid
      dict(name="stack_256_grid1024", kind="stack", num=256, side=32, epsilon=0.01,
           iterations=0, about=75),
      # a generative model's loss: divergence and gradient
      dict(name="divergence_4096x3500_d64", kind="divergence", cloud="gauss", n=4096, m=3500,
           d=64, epsilon=0.05, precision="auto", iterations=0, about=20),
      # gradients through the potentials
      dict(name="implicit_2000x1500_d8", kind="implicit", cloud="gauss", n=2000, m=1500, d=8,
           epsilon=0.1, precision="auto", iterations=0, about=20),
      # the plan applied to the points' coordinates and a weight (d + 2 vectors)
      dict(name="apply_16384x12001_d64_k66", kind="apply", cloud="gauss", n=16384, m=12001,
           d=64, k=66, axis=1, epsilon=0.05, precision="auto"),
  ]


def _log_size(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["solve"] * 6 + ["batch", "stack", "divergence", "implicit", "apply"])
  if kind == "batch":
    return dict(kind=kind, num=rng.randint(8, 96), lo=rng.choice([64, 128, 200]),
                hi=_log_size(rng, 500, 4096), d=rng.choice([8, 32, 48]),
                epsilon=rng.choice([10.0, 13.0, 20.0]), precision=rng.choice(["auto", "fp32"]),
                iterations=INNER * rng.randint(1, 4), about=0)
  if kind == "stack":
    return dict(kind=kind, num=_log_size(rng, 16, 512), side=rng.choice([16, 24, 28, 32]),
                epsilon=rng.choice([0.01, 0.02, 0.05]), iterations=INNER * rng.randint(2, 8),
                about=0)
  cloud = rng.choice(["uniform", "gauss"])
  d = rng.choice([2, 2, 3, 3, 5, 8]) if cloud == "uniform" else rng.choice(
      [10, 16, 24, 32, 50, 64, 64, 64, 96, 128])
  if kind == "solve":
    hi = 16000 if d < 32 else 24000
    decay = rng.choice([1.0, 1.0, 1.0, 0.8])
    return dict(kind=kind, cloud=cloud, n=_log_size(rng, 64, hi), m=_log_size(rng, 64, hi), d=d,
                epsilon=rng.choice([0.01, 0.02, 0.05, 0.1]), relative="mean",
                scale_cost=rng.choice(["", "", "mean"]), decay=decay,
                precision=rng.choice(["auto", "auto", "auto", "fp32"]),
                iterations=INNER * rng.randint(2, 6), about=0)
  if kind == "divergence":
    return dict(kind=kind, cloud=cloud, n=_log_size(rng, 200, 8192),
                m=_log_size(rng, 200, 8192), d=d, epsilon=rng.choice([0.05, 0.1]),
                precision="auto", iterations=INNER * rng.randint(1, 3), about=0)
  if kind == "implicit":
    return dict(kind=kind, cloud=cloud, n=_log_size(rng, 100, 2500),
                m=_log_size(rng, 100, 2500), d=min(d, 16), epsilon=rng.choice([0.1, 0.2]),
                precision="auto", iterations=INNER * rng.randint(2, 4), about=0)
  return dict(kind=kind, cloud=cloud, n=_log_size(rng, 200, 16384),
              m=_log_size(rng, 200, 16384), d=d, k=_log_size(rng, 1, 96), axis=rng.choice([0, 1]),
              epsilon=rng.choice([0.05, 0.1]), precision=rng.choice(["auto", "fp32"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
  return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _rand(g, *shape):
  return torch.rand(shape, generator=g, device="cuda")


def _randn(g, *shape):
  return torch.randn(shape, generator=g, device="cuda")


def _clouds(case, seed):
  """x, y, a, b: uniform clouds with uneven weights, or Gaussian clouds with
  a shift and uniform weights."""
  n, m, d = case["n"], case["m"], case["d"]
  g = _gen(seed)
  if case["cloud"] == "uniform":
    x, y = _rand(g, n, d), _rand(g, m, d)
    a, b = _rand(g, n) + 0.2, _rand(g, m) + 0.2
    return x, y, a / a.sum(), b / b.sum()
  x = _randn(g, n, d)
  var = 0.5 + 1.5 * _rand(g, d)
  y = 0.5 + _randn(g, m, d) * var.sqrt()
  return (x, y, torch.full((n,), 1.0 / n, device="cuda"), torch.full((m,), 1.0 / m, device="cuda"))


def _batch_sizes(case):
  r = random.Random(case["num"] * 1000 + case["hi"])
  lo, hi = math.log(case["lo"]), math.log(case["hi"])
  size = lambda: int(math.exp(r.uniform(lo, hi)))  # noqa: E731
  return [(size(), size()) for _ in range(case["num"])]


def _mixture(g, n, d):
  means = 2.0 * _randn(g, 4, d)
  comp = torch.randint(0, 4, (n,), generator=g, device="cuda")
  return means[comp] + 0.5 * _randn(g, n, d)


def _dirichlet(g, n):
  e = -torch.log1p(-_rand(g, n).clamp(max=1.0 - 1e-6)) + 1e-6
  return e / e.sum()


def _grid(side):
  t = torch.linspace(0.0, 1.0, side, device="cuda")
  gx, gy = torch.meshgrid(t, t, indexing="ij")
  return torch.stack([gx.reshape(-1), gy.reshape(-1)], 1).contiguous()


def _grid_weights(g, num, grid):
  """Mixtures of up to five Gaussians on the grid, with a floor."""
  mu, sd_, e = _rand(g, num, 5, 2), 0.03 + 0.17 * _rand(g, num, 5), _rand(g, num, 5)
  pi = e / e.sum(1, keepdim=True)
  d2 = ((grid[None, :, None, :] - mu[:, None]) ** 2).sum(-1)
  dens = ((pi / sd_ ** 2)[:, None] * torch.exp(-d2 / (2 * sd_ ** 2)[:, None])).sum(-1)
  w = dens / dens.sum(1, keepdim=True) + 1e-6
  return (w / w.sum(1, keepdim=True)).contiguous()


def _solver_kwargs(case):
  kw = dict(precision=case.get("precision", "auto"))
  if case["iterations"]:
    kw.update(min_iterations=case["iterations"], max_iterations=case["iterations"])
  return kw


def _geometry(case, x, y):
  """The geometry as a program builds it on new points."""
  kw = {}
  if case.get("scale_cost"):
    kw["scale_cost"] = case["scale_cost"]
  if case["epsilon"]:
    kw["epsilon"] = case["epsilon"]
  if case.get("relative", "mean"):
    kw["relative_epsilon"] = case.get("relative", "mean")
  geom = pointcloud.PointCloud(x, y, **kw)
  if case.get("decay", 1.0) < 1.0:
    sched = epsilon_scheduler.Epsilon(geom.epsilon, init=20.0, decay=case["decay"])
    geom = pointcloud.PointCloud(x, y, epsilon=sched, scale_cost=1.0 / geom.inv_scale_cost)
  return geom


def prepare(case, seed):
  kind = case["kind"]
  state = dict(case=case, kw=_solver_kwargs(case) if "iterations" in case else {})
  if kind == "batch":
    g = _gen(seed)
    state["x"], state["y"], state["a"], state["b"] = [], [], [], []
    for n, m in _batch_sizes(case):
      state["x"].append(_mixture(g, n, case["d"]))
      state["y"].append(_mixture(g, m, case["d"]))
      state["a"].append(_dirichlet(g, n))
      state["b"].append(_dirichlet(g, m))
  elif kind == "stack":
    grid = _grid(case["side"])
    w = _grid_weights(_gen(seed), 2 * case["num"], grid)
    state["geom"] = pointcloud.PointCloud(grid, epsilon=case["epsilon"])
    state["a"], state["b"] = w[0::2].contiguous(), w[1::2].contiguous()
    state["solver"] = sinkhorn.Sinkhorn(**state["kw"])
  else:
    state["x"], state["y"], state["a"], state["b"] = _clouds(case, seed)
    g = _gen(seed + 1000003)
    if kind == "implicit":
      n, m = case["n"], case["m"]
      w, v = _randn(g, n) / n, _randn(g, m) / m
      state["w"], state["v"] = w, v + (w.sum() - v.sum()) / m
    elif kind == "apply":
      f, gg, eps = _potentials64(case, state)
      state["f"], state["g"] = f.float(), gg.float()
      state["geom"] = pointcloud.PointCloud(state["x"], state["y"], epsilon=eps)
      state["vec"] = _randn(g, case["k"], case["n"] if case["axis"] == 0 else case["m"])
      if case["k"] == 1:
        state["vec"] = state["vec"][0].contiguous()
  return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
  case = state["case"]
  kind = case["kind"]
  if kind == "solve":
    out = linear.solve(_geometry(case, state["x"], state["y"]), state["a"], state["b"],
                       **state["kw"])
    return dict(f=out.f, g=out.g, errors=out.errors, cost=out.reg_ot_cost, n_iters=out.n_iters)
  if kind == "batch":
    geoms = [pointcloud.PointCloud(x, y, epsilon=case["epsilon"])
             for x, y in zip(state["x"], state["y"])]
    outs = linear.solve_batch(geoms, state["a"], state["b"], **state["kw"])
    return dict(f=torch.cat([o.f for o in outs]), g=torch.cat([o.g for o in outs]),
                cost=np.array([o.reg_ot_cost for o in outs], np.float32))
  if kind == "stack":
    out = sinkhorn.run_stacked(state["geom"], state["a"], state["b"], state["solver"])
    return dict(f=out.f, g=out.g, cost=out.reg_ot_cost.astype(np.float32))
  if kind == "divergence":
    x = state["x"].detach().requires_grad_()
    y = state["y"].detach().requires_grad_()
    div, out = sd.sinkhorn_divergence(pointcloud.PointCloud, x, y, a=state["a"], b=state["b"],
                                      epsilon=case["epsilon"], relative_epsilon="mean",
                                      solve_kwargs=state["kw"])
    div.backward()
    return dict(divergence=div.detach().float(), gx=x.grad, gy=y.grad,
                f=out.potentials[0][0].detach(), g=out.potentials[0][1].detach())
  if kind == "implicit":
    x = state["x"].detach().requires_grad_()
    y = state["y"].detach().requires_grad_()
    out = linear.solve(_geometry(case, x, y), state["a"], state["b"], **state["kw"])
    loss = (out.f * state["w"]).sum() + (out.g * state["v"]).sum()
    loss.backward()
    return dict(gx=x.grad, gy=y.grad, f=out.f.detach(), g=out.g.detach())
  return state["geom"].apply_transport_from_potentials(
      state["f"], state["g"], state["vec"], axis=case["axis"], precision=case["precision"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
  """Inputs read once, outputs written once; per cost entry of a sweep the
  inner product (2 d) and an exponential with its sum (4)."""
  kind = case["kind"]
  its = case.get("iterations") or case.get("about") or 0
  if kind == "batch":
    sizes, d = _batch_sizes(case), case["d"]
    pts = sum(n + m for n, m in sizes)
    ent = sum(n * m for n, m in sizes)
    return {"bytes": 4.0 * pts * (d + 2), "flops": ent * 2.0 * its * (2 * d + 4)}
  if kind == "stack":
    p = case["side"] ** 2
    return {"bytes": 16.0 * p * case["num"], "flops": 2.0 * its * case["num"] * p * p * 8.0}
  n, m, d = case["n"], case["m"], case["d"]
  pts, ent = n + m, float(n) * m
  if kind == "solve":
    return {"bytes": 4.0 * pts * (d + 2), "flops": 2.0 * its * ent * (2 * d + 4)}
  if kind == "divergence":
    sym = float(n) * n + float(m) * m
    fwd = its * (2.0 * ent + sym) * (2 * d + 4)
    return {"bytes": 4.0 * pts * (2 * d + 2), "flops": fwd + (2.0 * ent + sym) * (4 * d + 6)}
  if kind == "implicit":
    # the solve, a few plan products per side, the pullback's 2 (d + 1)
    # vectors on each side
    return {"bytes": 4.0 * pts * (2 * d + 4),
            "flops": ent * ((2.0 * its + 20) * (2 * d + 4) + 8.0 * (d + 1))}
  k = case["k"]
  return {"bytes": 4.0 * (pts * (d + 1) + k * pts), "flops": ent * (2.0 * d + 4 + 2 * k)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _mean_std(x, y):
  """mean(C) and std(C) of the unscaled cost, from moments."""
  nx, ny = (x * x).sum(1), (y * y).sum(1)
  mx, my = x.mean(0), y.mean(0)
  mean = nx.mean() + ny.mean() - 2.0 * (mx @ my)
  tr = ((x.t() @ x) * (y.t() @ y)).sum() / (x.shape[0] * y.shape[0])
  sq = ((nx ** 2).mean() + (ny ** 2).mean() + 2.0 * nx.mean() * ny.mean() + 4.0 * tr
        - 4.0 * ((nx[:, None] * x).mean(0) @ my) - 4.0 * ((ny[:, None] * y).mean(0) @ mx))
  return float(mean), math.sqrt(max(float(sq) - float(mean) ** 2, 0.0))


def _eps_inv(case, x, y):
  """epsilon and 1 / (scale of the cost), as the solver gets them (FP32)."""
  mean, std = _mean_std(x, y)
  inv = 1.0 / mean if case.get("scale_cost") == "mean" else 1.0
  if case.get("relative", "mean") == "mean":
    eps = case["epsilon"] * inv * mean
  else:
    eps = case["epsilon"] or 0.05 * inv * std
  return float(np.float32(eps)), float(np.float32(inv))


class _Cost:
  """Row and column log-sum-exps of ``(pot - C) / eps`` in blocks."""

  def __init__(self, x, y, inv):
    self.x, self.y, self.inv = x, y, inv
    self.nx, self.ny = inv * (x * x).sum(1), inv * (y * y).sum(1)
    self.step = max(1, int(1.5e8 // y.shape[0]))
    self.dense = None
    if x.shape[0] * y.shape[0] <= 3e8:
      self.dense = self.block(0, x.shape[0])

  def block(self, i, j):
    c = torch.addmm(self.ny[None], self.x[i:j], self.y.t(), alpha=-2.0 * self.inv)
    return c.add_(self.nx[i:j, None])

  def blocks(self):
    n = self.x.shape[0]
    for i in range(0, n, self.step):
      j = min(n, i + self.step)
      yield i, j, (self.dense[i:j] if self.dense is not None else self.block(i, j))

  def over_rows(self, f, eps):
    """eps LSE_i((f_i - C_ij) / eps), one per column."""
    run = None
    for i, j, c in self.blocks():
      part = torch.logsumexp((f[i:j, None] - c).div_(eps), 0)
      run = part if run is None else torch.logaddexp(run, part)
    return eps * run

  def over_cols(self, g, eps):
    out = torch.empty_like(self.nx)
    for i, j, c in self.blocks():
      out[i:j] = torch.logsumexp((g[None] - c).div_(eps), 1)
    return eps * out

  def plan(self, f, g, eps):
    for i, j, c in self.blocks():
      yield i, j, torch.exp((f[i:j, None] + g[None] - c) / eps)


def _solve64(case, x, y, a, b, eps, inv, symmetric=False):
  """The loop of the solver: blocks of INNER iterations, the error of the
  column marginal after each block, the stop test."""
  cost = _Cost(x, y, inv)
  fixed = case["iterations"]
  limit = fixed or MAX_ITERATIONS
  f, g = torch.zeros_like(a), torch.zeros_like(b)
  la, lb = torch.log(a), torch.log(b)
  errors = torch.full((int(math.ceil(limit / INNER)),), -1.0, dtype=torch.float64, device="cuda")
  decay = case.get("decay", 1.0)
  it = 0
  while it < limit:
    for _ in range(INNER):
      e = eps * max((20.0 if decay < 1.0 else 1.0) * decay ** it, 1.0)
      if symmetric:
        g = 0.5 * g + 0.5 * (e * lb - cost.over_rows(g, e))
        f = g
      else:
        g = e * lb - cost.over_rows(f, e)
        f = e * la - cost.over_cols(g, e)
      it += 1
    if fixed and it < limit:
      errors[it // INNER - 1] = float("inf")
      continue
    marg = torch.exp((cost.over_rows(f, eps) + g) / eps)
    err = float((marg - b).abs().sum()) * (2.0 if symmetric else 1.0)
    errors[it // INNER - 1] = err
    if not fixed and err < THRESHOLD:
      break
  reg = ((a * (f - eps * la)).sum() + (b * (g - eps * lb)).sum()
         + eps * (a.sum() * b.sum() - marg.sum()))
  return f, g, errors, float(reg), it, cost


def _potentials64(case, state, its=5):
  x, y = state["x"].double(), state["y"].double()
  eps = float(np.float32(case["epsilon"] * _mean_std(x, y)[0]))
  cost = _Cost(x, y, 1.0)
  la, lb = torch.log(state["a"].double()), torch.log(state["b"].double())
  f = torch.zeros_like(la)
  for _ in range(its):
    g = eps * lb - cost.over_rows(f, eps)
    f = eps * la - cost.over_cols(g, eps)
  return f, g, eps


def _cost_gradient(cost, x, y, f, g, eps):
  """d/dx and d/dy of the regularised cost with the potentials held fixed."""
  gx, gy = torch.zeros_like(x), torch.zeros_like(y)
  cols = torch.zeros_like(g)
  for i, j, p in cost.plan(f, g, eps):
    gx[i:j] = p.sum(1)[:, None] * x[i:j] - p @ y
    gy -= p.t() @ x[i:j]
    cols += p.sum(0)
  gy += cols[:, None] * y
  return 2.0 * cost.inv * gx, 2.0 * cost.inv * gy


def _implicit64(state, x, y, a, b, f, g, eps, cost):
  """Gradient of <w, f> + <v, g> by the first-order conditions' Jacobian at
  (f, g): the Schur system on the smaller side in its symmetric form, its
  null direction moved to 1, then the pullback to the points."""
  w, v = state["w"].double(), state["v"].double()
  p = torch.cat([q for _, _, q in cost.plan(f, g, eps)])
  swap = p.shape[0] > p.shape[1]
  r = p.t() if swap else p
  gs, gl = (v, w) if swap else (w, v)
  ms, ml = r.sum(1), r.sum(0)
  c = ms.rsqrt()
  k = c[:, None] * r * ml.rsqrt()[None]
  q = ms.sqrt() / ms.sqrt().norm()
  mat = torch.eye(r.shape[0], dtype=torch.float64, device="cuda") - k @ k.t() + q[:, None] * q
  res = gs - r @ (gl / ml)
  res = res - res.mean()
  rhs = c * res
  rhs = rhs - q * (q @ rhs)
  z = torch.linalg.solve(mat, rhs) / c
  z = z - (z @ ms) / (ms @ ms) * ms
  other = gl - r.t() @ (z / ms)
  la, lb = (-other, -z) if swap else (-z, -other)
  ma, mb = p.sum(1), p.sum(0)
  gc = -p * ((la / ma)[:, None] + (lb / mb)[None])
  gx = 2.0 * cost.inv * (gc.sum(1)[:, None] * x - gc @ y)
  gy = 2.0 * cost.inv * (gc.sum(0)[:, None] * y - gc.t() @ x)
  return gx, gy


def exact(case, seed):
  state = prepare(case, seed)
  kind = case["kind"]
  if kind == "batch":
    fs, gs, cs = [], [], []
    eps = float(np.float32(case["epsilon"]))
    for x, y, a, b in zip(state["x"], state["y"], state["a"], state["b"]):
      f, g, _, reg, _, _ = _solve64(case, x.double(), y.double(), a.double(), b.double(), eps, 1.0)
      fs.append(f)
      gs.append(g)
      cs.append(reg)
    return dict(f=torch.cat(fs), g=torch.cat(gs), cost=np.array(cs))
  if kind == "stack":
    x = _grid(case["side"]).double()
    c = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist") ** 2
    eps = float(np.float32(case["epsilon"]))
    fixed, limit = case["iterations"], case["iterations"] or MAX_ITERATIONS
    a, b = state["a"].double(), state["b"].double()
    la, lb = torch.log(a), torch.log(b)
    f, g = torch.zeros_like(a), torch.zeros_like(b)
    live = torch.arange(a.shape[0], device="cuda")
    cost = torch.zeros(a.shape[0], dtype=torch.float64, device="cuda")
    lse = lambda h: torch.cat([  # noqa: E731
        torch.logsumexp((h[i:i + 64, None, :] - c[None]) / eps, 2)
        for i in range(0, h.shape[0], 64)]) * eps
    it = 0
    while it < limit and live.numel():
      fl, gl = f[live], g[live]
      for _ in range(INNER):
        gl = eps * lb[live] - lse(fl)
        fl = eps * la[live] - lse(gl)
      it += INNER
      f[live], g[live] = fl, gl
      if fixed and it < limit:
        continue
      marg = torch.exp((lse(fl) + gl) / eps)
      err = (marg - b[live]).abs().sum(1)
      al, bl = a[live], b[live]
      cost[live] = ((al * (fl - eps * la[live])).sum(1) + (bl * (gl - eps * lb[live])).sum(1)
                    + eps * (al.sum(1) * bl.sum(1) - marg.sum(1)))
      live = live[:0] if fixed else live[err >= THRESHOLD]
    return dict(f=f, g=g, cost=cost)
  x, y = state["x"].double(), state["y"].double()
  a, b = state["a"].double(), state["b"].double()
  if kind == "apply":
    eps, vec = float(state["geom"].epsilon), state["vec"].double()
    f, g = state["f"].double(), state["g"].double()
    cost, one = _Cost(x, y, 1.0), vec.ndim == 1
    vec = vec[None] if one else vec
    if case["axis"] == 1:
      out = torch.cat([p @ vec.t() for _, _, p in cost.plan(f, g, eps)]).t().contiguous()
    else:
      out = sum(vec[:, i:j] @ p for i, j, p in cost.plan(f, g, eps))
    return out[0] if one else out
  eps, inv = _eps_inv(case, x, y)
  f, g, errors, reg, its, cost = _solve64(case, x, y, a, b, eps, inv)
  if kind == "solve":
    return dict(f=f, g=g, errors=errors, cost=reg, n_iters=None)
  if kind == "divergence":
    gx, gy = _cost_gradient(cost, x, y, f, g, eps)
    div = reg
    for pts, wts, grad in ((x, a, gx), (y, b, gy)):
      fs, gs, _, r, _, cs = _solve64(case, pts, pts, wts, wts, eps, inv, symmetric=True)
      gl, gr = _cost_gradient(cs, pts, pts, fs, gs, eps)
      grad -= 0.5 * (gl + gr)
      div -= 0.5 * r
    div += 0.5 * eps * (float(a.sum()) - float(b.sum())) ** 2
    return dict(divergence=torch.tensor(div, dtype=torch.float64), gx=gx, gy=gy, f=f, g=g)
  gx, gy = _implicit64(state, x, y, a, b, f, g, eps, cost)
  return dict(gx=gx, gy=gy, f=f, g=g)
