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


@pytest.mark.parametrize("m,n,kk", [(40, 128, 512), (304, 264, 200), (2560, 2816, 128)])   # few rows, tiles, CTA pairs
@pytest.mark.parametrize("mn", [False, True])
def test_gemm_scaled_on_the_device(cuda_lib, m, n, kk, mn):
  """The factor in device memory multiplies the fp32 sums: the same bits as scaling an fp32 result and rounding."""
  torch.manual_seed(m)
  a, b = (torch.randn(*((kk, r) if mn else (r, kk)), device="cuda", dtype=torch.bfloat16) for r in (m, n))
  s = torch.tensor(-0.37, device="cuda")
  want = (k.gemm(a, b, a_mn=mn, b_mn=mn, epi=k.EPI_F32) * s).to(torch.bfloat16)
  assert torch.equal(k.gemm(a, b, a_mn=mn, b_mn=mn, scale=s), want)


@pytest.mark.parametrize("wanted", ["both", "weight", "hidden"])
def test_head_in_one_piece(cuda_lib, wanted):
  """All rows in one chunk: the weight gradient is made in the backward pass, as often as it is asked for."""
  h = torch.randn(1, 130, 64, device="cuda", dtype=torch.bfloat16, requires_grad=wanted != "weight")
  w = (torch.randn(520, 64, device="cuda") / 8).to(torch.bfloat16).requires_grad_(wanted != "hidden")
  t = torch.randint(0, 520, (1, 130), device="cuda")
  t[0, 3:50] = -100
  inputs = [x for x in (h, w) if x.requires_grad]
  loss = ops.linear_cross_entropy(h, w, t)
  first = torch.autograd.grad(loss, inputs, retain_graph=True)
  again = torch.autograd.grad(loss * 2, inputs)
  ref_in = [x.detach().double().requires_grad_(x.requires_grad) for x in (h, w)]
  want = torch.autograd.grad(F.cross_entropy((ref_in[0] @ ref_in[1].t())[0], t[0]), [x for x in ref_in if x.requires_grad])
  for a, b, r in zip(first, again, want):
    assert torch.equal(2 * a, b)
    assert ((a.double() - r).norm() / r.norm()).item() < 1e-2      # bf16 logits and bf16 d(logits)


@pytest.mark.parametrize("vocab", [8, 16376, 16384, 16392, 49160])
def test_cross_entropy_at_the_edges_of_its_loops(cuda_lib, vocab):
  logits = (3 * torch.randn(5, vocab, device="cuda")).to(torch.bfloat16)
  logits[1, :vocab // 2] = float("-inf")
  t = torch.tensor([0, vocab - 1, -100, vocab // 2, vocab - 8], device="cuda")
  x = logits.double().requires_grad_(True)
  want = F.cross_entropy(x, t, ignore_index=-100, reduction="sum")
  want.backward()
  loss = torch.zeros(1, device="cuda")
  k.ce_fwd_bwd_(logits, t, loss, torch.tensor([0.5], device="cuda"))
  assert abs(loss.item() / want.item() - 1) < 1e-5
  # bf16 results: 2^-9 of each value
  assert ((logits.double() - 0.5 * x.grad).abs() <= 2.0 ** -8 * (0.5 * x.grad).abs() + 1e-9).all()


@pytest.mark.parametrize("rows", [2048, 4096, 4097])
def test_memory_that_a_head_takes(cuda_lib, rows):
  """Up to 2 * hidden rows d(logits) are held instead of an fp32 weight gradient, above that 2048 rows beside it."""
  from torchprime_b200.models.llama import CausalLMHead
  hidden, vocab = 2048, 32768
  w = (torch.randn(vocab, hidden, device="cuda") / 32).to(torch.bfloat16).requires_grad_(True)
  h = torch.randn(1, rows, hidden, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  t = torch.randint(0, vocab, (1, rows), device="cuda")
  head = CausalLMHead.__new__(CausalLMHead)
  torch.nn.Module.__init__(head)
  head.norm, head.lm_head, head.loss_group = torch.nn.Identity(), torch.nn.Linear(1, 1, bias=False), None
  head.lm_head.weight = torch.nn.Parameter(w.detach())
  torch.cuda.synchronize()
  torch.cuda.reset_peak_memory_stats()
  before = torch.cuda.memory_allocated()
  loss = head(h, t, want_logits=False)[1]
  torch.cuda.synchronize()
  taken = torch.cuda.max_memory_allocated() - before
  held = 2 * rows * vocab if rows <= 2 * hidden else 4 * hidden * vocab + 2 * 2048 * vocab
  assert taken <= held + 2 * rows * hidden + (4 << 20)      # and the gradient of the hidden states, a few small tensors
  loss.backward()
  assert head.lm_head.weight.grad.dtype == torch.bfloat16 and bool(torch.isfinite(h.grad).all())
