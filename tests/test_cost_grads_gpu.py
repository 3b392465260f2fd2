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
