"""Router logits in fp32 and the gradient of the routing weights."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import functional as ops
from torchprime_b200.ops import moe


@pytest.mark.parametrize("E,K", [(8, 2), (33, 3), (64, 6), (256, 8), (5, 5), (4, 1)])
@pytest.mark.parametrize("mode", ["softmax", "sigmoid"])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_backward(cuda_lib, E, K, mode, norm, dtype):
  """Weights and scores both carry gradients; fp64 autograd through the same choice is the oracle."""
  torch.manual_seed(E)
  lg = torch.randn(77, E, device="cuda").to(dtype).requires_grad_(True)
  w, idx, sc = moe.router_topk(lg, K, mode=mode, norm_topk=norm, scale=1.7)
  gw, gs = torch.randn_like(w), torch.randn_like(sc)
  x = lg.detach().double().requires_grad_(True)
  s = torch.softmax(x, -1) if mode == "softmax" else torch.sigmoid(x)
  wr = s.gather(1, idx.long())
  if norm:
    wr = wr / wr.sum(-1, keepdim=True)
  wr = wr * 1.7
  tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6
  for outs, refs, grads in (([w, sc], [wr, s], [gw, gs]), ([w], [wr], [gw]), ([sc], [s], [gs])):
    (got,) = torch.autograd.grad(outs, lg, grads, retain_graph=True)
    (want,) = torch.autograd.grad(refs, x, [g.double() for g in grads], retain_graph=True)
    assert got.dtype == dtype
    assert bool(((got.double() - want).abs() <= tol * want.abs() + 5e-6).all()), (got - want).abs().max()


def test_linear_f32_gradients(cuda_lib):
  x = torch.randn(50, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  w = torch.randn(64, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  y = ops.linear_f32(x, w)
  assert y.dtype == torch.float32
  dy = torch.randn_like(y)
  dx, dw = torch.autograd.grad(y, (x, w), dy)
  assert torch.equal(dx, (dy @ w.float()).to(torch.bfloat16)) and torch.equal(dw, (dy.t() @ x.float()).to(torch.bfloat16))


@pytest.mark.parametrize("T,N,K", [(256, 64, 2048), (257, 8, 64), (1500, 64, 136), (300, 65, 1032), (1031, 256, 512), (4000, 120, 200)])
def test_linear_f32_gradient_kernels(cuda_lib, T, N, K):
  """Edges of rows, experts and columns; a view of wider rows; sums are fp32 ones (T or N terms) rounded to bf16 once."""
  torch.manual_seed(T)
  x = torch.randn(T, K + 8, device="cuda").bfloat16()[:, :K].requires_grad_(True)
  w = torch.randn(N, K, device="cuda").bfloat16().requires_grad_(True)
  dy = torch.randn(T, N, device="cuda")
  dx, dw = torch.autograd.grad(ops.linear_f32(x, w), (x, w), dy)
  for got, a, b in ((dx, dy.double(), w.detach().double()), (dw, dy.double().t(), x.detach().double())):
    want, size = a @ b, a.abs() @ b.abs()
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * size).all())
  (only,) = torch.autograd.grad(ops.linear_f32(x, w.detach()), x, dy)
  assert torch.equal(only, dx)


def test_linear_f32_gradient_of_a_gradient(cuda_lib):
  x = torch.randn(300, 64, device="cuda").bfloat16().requires_grad_(True)
  w = torch.randn(16, 64, device="cuda").bfloat16().requires_grad_(True)
  dy = torch.randn(300, 16, device="cuda", requires_grad=True)
  (dx,) = torch.autograd.grad(ops.linear_f32(x, w), x, dy, create_graph=True)
  ddy, dw = torch.autograd.grad(dx.float().square().sum(), (dy, w))
  assert ddy.shape == dy.shape and dw.abs().sum() > 0
  many = torch.autograd.grad(ops.linear_f32(x, w), x, torch.stack([dy, 2 * dy]).detach(), is_grads_batched=True)[0]
  assert torch.equal(many[0], (dy @ w.float()).to(torch.bfloat16))


@pytest.mark.parametrize("E,K", [(8, 2), (64, 6), (256, 8)])
@pytest.mark.parametrize("mode", ["softmax", "sigmoid"])
@pytest.mark.parametrize("norm", [True, False])
def test_router_backward_rounds_like_fp32(cuda_lib, E, K, mode, norm):
  """Wide logits, where a fast exponential is tens of ulp off.  Scores, W, the selected experts' terms and the products
  are fp32: each is off by a few roundings of the terms that are added (16 ulp of the larger side)."""
  torch.manual_seed(E)
  lg = (torch.randn(200, E, device="cuda") * 12).requires_grad_(True)
  w, idx, sc = moe.router_topk(lg, K, mode=mode, norm_topk=norm)
  gw, gs = torch.randn_like(w), torch.randn_like(sc)
  x = lg.detach().double().requires_grad_(True)
  s = torch.softmax(x, -1) if mode == "softmax" else torch.sigmoid(x)
  sel = s.gather(1, idx.long())
  total = sel.sum(-1, keepdim=True) if norm else torch.ones_like(sel[:, :1])
  (got,) = torch.autograd.grad([w, sc], lg, [gw, gs])
  (want,) = torch.autograd.grad([sel / total, s], x, [gw.double(), gs.double()])
  # |ds| of every expert, with the terms of the normalisation taken at their size and not at their difference
  c = (gw.double().abs() * sel).sum(-1, keepdim=True) / total if norm else 0.0
  ds = gs.double().abs().scatter_add(1, idx.long(), (gw.double().abs() + c) / total)
  size = s * (ds + (s * ds).sum(-1, keepdim=True)) if mode == "softmax" else s * ds
  err = ((got.double() - want).abs() / (size.detach() + 1e-30))
  assert err.max().item() < 16 * 2.0 ** -23, err.max().item() * 2.0 ** 23


@pytest.mark.parametrize("mode", ["softmax", "sigmoid"])
@pytest.mark.parametrize("norm", [True, False])
def test_router_batched_gradients(cuda_lib, mode, norm):
  """Several gradients in one backward pass give what one pass each gives (fp32 both ways: a few roundings apart)."""
  torch.manual_seed(1)
  lg = torch.randn(30, 16, device="cuda", requires_grad=True)
  w, _, sc = moe.router_topk(lg, 4, mode=mode, norm_topk=norm, scale=1.5)
  gw, gs = torch.randn(3, *w.shape, device="cuda"), torch.randn(3, *sc.shape, device="cuda")
  for outs, grads in (([w, sc], [gw, gs]), ([w], [gw]), ([sc], [gs])):
    (got,) = torch.autograd.grad(outs, lg, grads, is_grads_batched=True, retain_graph=True)
    for i in range(3):
      (one,) = torch.autograd.grad(outs, lg, [g[i] for g in grads], retain_graph=True)
      assert torch.allclose(got[i], one, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("E,K,groups", [(64, 6, 1), (256, 8, 8), (33, 3, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_takes_a_bf16_bias(cuda_lib, E, K, groups, dtype):
  """As a model keeps it: the same choices and weights as with its fp32 copy, native and from Python."""
  torch.manual_seed(E)
  lg, bias = torch.randn(77, E, device="cuda").to(dtype), (0.3 * torch.randn(E, device="cuda")).bfloat16()
  args = (K, 1, groups, max(1, groups // 2), True, 2.5)
  want = moe._router_forward(lg, bias.float(), *args)
  with torch.no_grad():
    native = ops._native().router_topk(lg, bias, *args)
  for got in (moe._router_forward(lg, bias, *args), native):
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_linear_f32_gradients_of_very_many_rows(cuda_lib):
  """One row more than a grid's second dimension has blocks of 64."""
  t, n, kk = 64 * 65535 + 1, 48, 8
  x = torch.randn(t, kk, device="cuda").bfloat16().requires_grad_(True)
  w = torch.randn(n, kk, device="cuda").bfloat16().requires_grad_(True)
  dy = torch.randn(1, n, device="cuda").expand(t, n)
  dx, dw = torch.autograd.grad(ops.linear_f32(x, w), (x, w), dy)
  one = (dy[:1].double() @ w.detach().double())
  assert bool(((dx.double() - one).abs() <= 2 ** -8 * one.abs() + 1e-5).all())
  want = dy[0].double()[:, None] * x.detach().double().sum(0)
  size = dy[0].double().abs()[:, None] * x.detach().double().abs().sum(0)
  assert bool(((dw.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * size).all())


@pytest.mark.parametrize("give_back", ["columns first", "elsewhere", "unaligned", "wider"])
def test_linear_f32_gradients_with_saved_tensor_hooks(cuda_lib, give_back):
  """Hooks may give saved tensors back in another layout, alignment or type; torch's operators take them as they are."""
  torch.manual_seed(1)
  x = torch.randn(300, 64, device="cuda").bfloat16().requires_grad_(True)
  w = torch.randn(16, 64, device="cuda").bfloat16().requires_grad_(True)
  dy = torch.randn(300, 16, device="cuda")

  def back(t):
    if give_back == "columns first":
      return t.t().contiguous().t()
    if give_back == "unaligned":
      return torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape)
    return t.float() if give_back == "wider" else t.clone()

  with torch.autograd.graph.saved_tensors_hooks(lambda t: t, back):
    y = ops.linear_f32(x, w)
    dx, dw = torch.autograd.grad(y, (x, w), dy)
  for got, a, b in ((dx, dy.double(), w.detach().double()), (dw, dy.double().t(), x.detach().double())):
    want, size = a @ b, a.abs() @ b.abs()
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * size).all())


@pytest.mark.parametrize("T,N,K,dx_kernel,dw_kernel", [
  (255, 64, 2048, False, False), (256, 64, 2048, True, True), (4096, 64, 2048, True, True), (4096, 8, 512, True, True),
  (4097, 8, 512, False, False), (5000, 16, 1024, False, False), (8192, 24, 512, True, True), (8200, 32, 2048, False, False),
  (9000, 40, 1024, True, False), (9000, 48, 2048, True, True), (256, 128, 4096, True, False), (260, 128, 4096, False, False),
  (1500, 128, 2048, False, True), (4097, 160, 512, False, False), (700, 256, 1024, False, True), (700, 256, 2048, False, False),
  (300, 512, 512, False, False)])
def test_logit_gradients_by_rule(cuda_lib, monkeypatch, T, N, K, dx_kernel, dw_kernel):
  """Each gradient comes from the kernel where that is the faster one, and is the same operators' bits as ever elsewhere."""
  from torchprime_b200.ops import kernels as k
  torch.manual_seed(T)
  asked = [False, False]
  kernel = k.linear_f32_bwd
  monkeypatch.setattr(k, "linear_f32_bwd", lambda dy, x, w, a=True, b=True: (asked.__setitem__(slice(None), [a, b]), kernel(dy, x, w, a, b))[1])
  x = torch.randn(T, K, device="cuda").bfloat16().requires_grad_(True)
  w = torch.randn(N, K, device="cuda").bfloat16().requires_grad_(True)
  dy = torch.randn(T, N, device="cuda")
  dx, dw = torch.autograd.grad(ops.linear_f32(x, w), (x, w), dy)
  assert asked == [dx_kernel, dw_kernel]
  for got, by_kernel, a, b, lib in ((dx, dx_kernel, dy.double(), w.detach().double(), (dy @ w.float()).to(torch.bfloat16)),
                                    (dw, dw_kernel, dy.double().t(), x.detach().double(), (dy.t() @ x.float()).to(torch.bfloat16))):
    want, size = a @ b, a.abs() @ b.abs()
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * size).all())
    assert by_kernel or torch.equal(got, lib)
  (only,) = torch.autograd.grad(ops.linear_f32(x, w.detach()), x, dy)
  assert torch.equal(only, dx)
