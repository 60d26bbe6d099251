"""Input gradient of a grouped gate / up projection as one contraction."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import moe


@pytest.mark.parametrize("e,f", [(3, 64), (4, 192), (2, 1024), (3, 72)])
def test_input_gradient_over_gate_and_up(cuda_lib, e, f):
  """One contraction over [dgate | dup]; f = 72 keeps the two-pass form."""
  torch.manual_seed(f)
  idx = torch.randint(0, e, (150, 2), device="cuda", dtype=torch.int32)
  plan = moe.build_dispatch_plan(idx, e)
  dgu = torch.randn(plan.num_rows, 2 * f, device="cuda", dtype=torch.bfloat16) * (plan.src_row >= 0)[:, None]
  wg, wu = ((torch.randn(e, 128, f, device="cuda") / f ** 0.5).to(torch.bfloat16) for _ in range(2))
  got = moe.grouped_dgrad_gate_up(dgu, wg, wu, plan)
  off = plan.k_offsets.tolist()
  for x in range(e):
    d = dgu[off[x]:off[x + 1]].double()
    want = d[:, :f] @ wg[x].double().t() + d[:, f:] @ wu[x].double().t()
    assert bool(((got[off[x]:off[x + 1]].double() - want).abs() <= 2.0 ** -6 * want.abs() + 0.02).all())
