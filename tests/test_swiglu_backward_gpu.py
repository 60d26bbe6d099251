"""The gradient of silu(g) * u inside the down projection's input gradient (TPB_EPI_SWIGLU_BWD) and the MLP as one node."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import _lib, functional as ops, kernels as k, moe

BF = torch.bfloat16


def _want(dact, gu):
  g, u = gu.double().chunk(2, -1)
  s = torch.sigmoid(g)
  return torch.cat([dact * u * (s + g * s * (1 - s)), dact * g * s], -1)


def _check(got, want, scale):
  # one bf16 rounding of fp32 values; `scale`: what the fp32 sums behind them carry
  assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + scale).all()), (got.double() - want).abs().max()


# edges of the 128 / 256-row tiles, columns that end inside a tile, a box and a half, few tiles and CTA pairs
@pytest.mark.parametrize("m,f,d", [(129, 8, 64), (200, 72, 136), (300, 264, 192), (2304, 2112, 64)])
@pytest.mark.parametrize("b_mn", [True, False])
def test_dense(cuda_lib, m, f, d, b_mn):
  torch.manual_seed(m)
  dy, w = torch.randn(m, d, device="cuda").to(BF), (torch.randn(d, f, device="cuda") / d ** 0.5).to(BF)
  gu = torch.randn(m, 2 * f, device="cuda").to(BF)
  big = torch.full((m + 2, 2 * f + 16), 5.0, device="cuda", dtype=BF)
  out = big[1:m + 1, 8:2 * f + 8]
  k.gemm(dy, w if b_mn else w.t().contiguous(), b_mn=b_mn, epi=k.EPI_SWIGLU_BWD, aux=gu, out=out)
  _check(out, _want(dy.double() @ w.double(), gu), 1e-5 * 8)
  out.fill_(5.0)
  assert bool((big == 5.0).all())


@pytest.mark.parametrize("align", [128, 256])
@pytest.mark.parametrize("f", [64, 328])
def test_grouped(cuda_lib, align, f):
  torch.manual_seed(f)
  e, d = 5, 64
  idx = torch.randint(0, e - 1, (300, 2), device="cuda", dtype=torch.int32)
  plan = moe.build_dispatch_plan(idx, e, row_align=align)
  live = (plan.src_row >= 0)[:, None]
  dy, gu = torch.randn(plan.num_rows, d, device="cuda").to(BF) * live, torch.randn(plan.num_rows, 2 * f, device="cuda").to(BF) * live
  w = (torch.randn(e, f, d, device="cuda") / d ** 0.5).to(BF)
  got = moe.grouped_gemm_rows(dy, w, plan, b_mn=False, epi=_lib.EPI_SWIGLU_BWD, c2=gu)
  off = plan.k_offsets.tolist()
  for x in range(e):
    r = slice(off[x], off[x + 1])
    _check(got[r], _want(dy[r].double() @ w[x].double().t(), gu[r]), 1e-5 * 8)


def test_extremes_of_the_gate(cuda_lib):
  """Gates whose sigmoid is 0 or 1 to the last bit, infinities and zeros, as in the kernel of its own."""
  g = torch.tensor([0.0, -0.0, 90.0, -90.0, 3e38, -3e38, float("inf"), 1e-30], device="cuda").to(BF)
  gu = torch.cat([g.repeat(160, 1), torch.full((160, 8), 0.5, device="cuda", dtype=BF)], -1)
  dy, w = torch.ones(160, 64, device="cuda", dtype=BF), torch.eye(64, 8, device="cuda").to(BF)
  got = k.gemm(dy, w, b_mn=True, epi=k.EPI_SWIGLU_BWD, aux=gu)
  want = k.swiglu_bwd(k.gemm(dy, w, b_mn=True), gu)
  assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))


@pytest.mark.parametrize("rows", [1, 128, 129, 400])
@pytest.mark.parametrize("grads", [(1, 1, 1, 1, 1), (1, 0, 0, 0, 0), (0, 1, 0, 0, 0), (0, 0, 0, 1, 1), (1, 1, 1, 0, 0)])
def test_mlp_as_one_node(cuda_lib, rows, grads, monkeypatch):
  """Against the two operators it stands for: the same result, gradients but for one rounding less."""
  _lib.lib()
  g = torch.Generator("cuda").manual_seed(rows)
  r = lambda *s: torch.randn(*s, device="cuda", generator=g)    # noqa: E731
  x, flat, wd, res = r(1, rows, 64).to(BF), (r(2 * 72, 64) / 8).to(BF), (r(64, 72) / 8).to(BF), r(1, rows, 64).to(BF)
  dy = r(1, rows, 64).to(BF)
  def call(fn):
    ts = [x.clone(), flat[:72].detach(), flat[72:].detach(), wd.clone(), res.clone()]
    for t, on in zip(ts, grads):
      t.requires_grad_(bool(on))
    y = fn(*ts)
    return [y.detach()] + list(torch.autograd.grad(y, [t for t in ts if t.requires_grad], dy))
  got = call(ops.swiglu_mlp)
  want = call(lambda x, a, b, c, res: ops.linear(ops.linear_swiglu(x, a, b), c, residual=res))
  assert torch.equal(got[0], want[0])
  for a, b in zip(got[1:], want[1:]):
    assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 5e-3     # bf16 gradient of the activation
  monkeypatch.setattr(_lib, "_native", None)
  for a, b in zip(call(ops.swiglu_mlp), want):
    assert torch.equal(a, b)


class _Published:
  """A gather whose shards have all landed."""
  world, epoch = 1, 1

  def __init__(self, flat):
    self.flat, self.base, self.shard_elems, self.chunk_elems = flat, flat.data_ptr(), flat.numel(), 4096
    self.flags = torch.ones((flat.numel() + 4095) // 4096, device="cuda", dtype=torch.int32)

  def offset_of(self, w):
    return (w.data_ptr() - self.base) // 2

  def wait_all(self):
    pass


# few rows, a few-rows product and a tiled one behind it; `grads` as above without the residual's
@pytest.mark.parametrize("rows", [40, 129, 400])
@pytest.mark.parametrize("grads", [(1, 1, 1, 1), (0, 1, 1, 1), (1, 0, 0, 1)])
@pytest.mark.parametrize("sink", [torch.float32, BF])
@pytest.mark.parametrize("gather", [False, True])
def test_mlp_whose_weights_collect_their_gradients(cuda_lib, rows, grads, sink, gather, monkeypatch):
  """The same node where gradients go to a main_grad, first overwritten and then added to, also while the weights are
  being gathered: the result of the two operators, gradients but for one rounding less."""
  g = torch.Generator("cuda").manual_seed(rows)
  r = lambda *s: torch.randn(*s, device="cuda", generator=g)    # noqa: E731
  flat = (torch.cat([r(2 * 72 * 64), r(64 * 72)]) / 8).to(BF)
  x, res, dy = r(1, rows, 64).to(BF), r(1, rows, 64).to(BF), r(1, rows, 64).to(BF)

  def call(fn):
    mains = torch.full((flat.numel(),), 3.0, device="cuda", dtype=sink)
    xs, rs = x.clone().requires_grad_(bool(grads[0])), res.clone().requires_grad_(True)
    ws, at = [], 0
    for (a, b), on in zip(((72, 64), (72, 64), (64, 72)), grads[1:]):
      w = flat[at:at + a * b].view(a, b).detach().requires_grad_(bool(on))
      w.main_grad, w.grad_overwrite = mains[at:at + a * b].view(a, b), True
      ws.append(w)
      at += a * b
    out = []
    for _ in range(2):
      ops.set_gather_context(_Published(flat) if gather else None)
      try:
        y = fn(xs, *ws, rs)
      finally:
        ops.set_gather_context(None)
      y.backward(dy)
      out += [y.detach(), mains.clone()]
    assert all(w.grad is None for w in ws)
    return out + [t.grad for t in (xs, rs) if t.requires_grad], type(y.grad_fn).__name__

  got, node = call(ops.swiglu_mlp)
  want, _ = call(lambda x, a, b, c, res: ops.linear(ops.linear_swiglu(x, a, b), c, residual=res))
  assert node == "_SwigluMlpFnBackward"
  assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
  for a, b in zip(got, want):
    assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 5e-3     # bf16 gradient of the activation
