"""ottb_reg_ot_cost_grads against the same formula in float64 tensor
operations on the same plan applications, at the edges of its 32 x 32 tiles.
Both compute in FP64 from the same FP32 inputs in the same order, up to the
order of the weights' sums: 1e-12 relative; a float32 output adds one
rounding."""
import numpy as np
import pytest

from tests import helpers, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,d", [(1, 1, 1), (31, 33, 2), (32, 64, 31), (65, 32, 32), (40, 50, 33),
                                   (129, 97, 64), (70, 60, 128)])
def test_matches_tensor_formula(n, m, d):
  import torch
  x, y, a, b = problems.uniform_cloud_problem(n, m, d, seed=n + d)
  if n > 3:
    a[1] = 0  # a zero weight's gradient is eps sum(b) alone
    a = (a / a.sum()).astype(np.float32)
  _, out = helpers.gpu_solve(x, y, a, b, epsilon=0.3)
  want = out._reg_ot_cost_grads()
  got = out.reg_ot_cost_grads()
  for w, g in zip(want, got):
    assert g.dtype == torch.float64 and g.shape == w.shape
    scale = max(float(w.abs().max()), 1e-30)
    assert float((g - w).abs().max()) <= 1e-12 * scale
  # a scale, float32 outputs, only some of the gradients
  s = torch.tensor(-0.75, dtype=torch.float64, device="cuda")
  for need in ((True, False, False, True), (False, True, True, False)):
    part = out._fixed_potential_grads(need, s, torch.float32)
    for flag, w, g in zip(need, want, part):
      if not flag:
        assert g is None
        continue
      assert g.dtype == torch.float32
      ref = -0.75 * w
      assert float((g.double() - ref).abs().max()) <= 2.0 ** -23 * max(float(ref.abs().max()), 1e-30)


def test_batched_grad_outputs():
  """is_grads_batched and a vectorized jacobian: the scaled gradients, each
  with one float32 rounding, as one call after another."""
  import torch
  from ott_b200.geometry import pointcloud
  from ott_b200.solvers import linear
  x, y, a, b = (torch.as_tensor(t).cuda() for t in problems.uniform_cloud_problem(40, 50, 3, seed=1))
  x.requires_grad_()
  a.requires_grad_()
  cost = lambda x: linear.reg_ot_cost(pointcloud.PointCloud(x, y, epsilon=0.1), a, b)  # noqa: E731
  c = cost(x)
  scales = torch.tensor([1.0, -2.0, 3.0], dtype=torch.float64, device="cuda")
  batched = torch.autograd.grad(c, [x, a], grad_outputs=scales, is_grads_batched=True,
                                retain_graph=True)
  for k, s in enumerate(scales):
    one = torch.autograd.grad(c, [x, a], grad_outputs=s, retain_graph=True)
    for got, want in zip(batched, one):
      bound = 2.0 ** -23 * float(want.abs().max())
      assert float((got[k] - want).abs().max()) <= bound
  two = lambda x: torch.stack([cost(x), 2 * cost(x)])  # noqa: E731
  jac = torch.autograd.functional.jacobian
  want = jac(two, x)
  assert float((jac(two, x, vectorize=True) - want).abs().max()) <= \
      2.0 ** -23 * float(want.abs().max())


def test_potentials_of_another_length():
  """Refused, as the tensor formula's arithmetic refuses them, before a
  kernel reads them."""
  import torch
  x, y, a, b = problems.uniform_cloud_problem(40, 50, 3, seed=1)
  _, out = helpers.gpu_solve(x, y, a, b, epsilon=0.3)
  for wrong in ((out.f[:-1], out.g), (out.f, torch.cat([out.g, out.g]))):
    with pytest.raises(ValueError):
      out._replace(potentials=wrong).reg_ot_cost_grads()
