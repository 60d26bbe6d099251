"""Weight gradient of the chunked head: fp32 over the chunks, delivered in one pass."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import functional as ops
from torchprime_b200.ops import kernels as k


@pytest.mark.parametrize("n", [8, 1000, 8 * 12345])
@pytest.mark.parametrize("scale", [1.0, -0.37, 0.0])
def test_scale_cast(cuda_lib, n, scale):
  x = torch.randn(n, device="cuda")
  s = torch.tensor(scale, device="cuda")
  assert torch.equal(k.scale_cast_bf16(x, s), (x * s).to(torch.bfloat16))


@pytest.mark.parametrize("rows,chunk", [(1, 64), (64, 64), (65, 64), (200, 64)])
def test_head_gradient_over_chunks(cuda_lib, rows, chunk):
  """The first chunk overwrites the fp32 weight gradient, the others add to it."""
  torch.manual_seed(rows)
  h = torch.randn(1, rows, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  w = (torch.randn(512, 64, device="cuda") / 8).to(torch.bfloat16).requires_grad_(True)
  t = torch.randint(0, 512, (1, rows), device="cuda")
  (2.5 * ops.linear_cross_entropy(h, w, t, chunk_rows=chunk)).backward()
  hd, wd = h.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
  (2.5 * F.cross_entropy((hd @ wd.t())[0], t[0])).backward()
  for got, want in ((h.grad, hd.grad), (w.grad, wd.grad)):
    assert ((got.double() - want).norm() / want.norm()).item() < 1e-2      # bf16 logits and bf16 d(logits)


def test_batched_gradients(cuda_lib):
  """Several gradients in one backward pass give what one pass each gives."""
  h = torch.randn(1, 70, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  w = (torch.randn(512, 64, device="cuda") / 8).to(torch.bfloat16).requires_grad_(True)
  loss = ops.linear_cross_entropy(h, w, torch.randint(0, 512, (1, 70), device="cuda"))
  scales = torch.tensor([1.0, -0.5, 3.0], device="cuda", dtype=loss.dtype)
  got = torch.autograd.grad(loss, (h, w), scales, is_grads_batched=True, retain_graph=True)
  for i in range(3):
    for a, b in zip(got, torch.autograd.grad(loss, (h, w), scales[i], retain_graph=True)):
      assert torch.equal(a[i], b)
