"""Attention backward for query / key head dim 192 and value dim 128 against the fp32 definition."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import attention_sm100 as A
from torchprime_b200.ops import reference as ref


def _check(b, sq, sk, hq, hkv, bound=2e-2, **kw):
  """The bound is that of the head-dim-128 tests (bf16 P and dS)."""
  torch.manual_seed(sq + sk)
  q, k, v = (torch.randn(b, s, h, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
             for s, h, d in ((sq, hq, 192), (sk, hkv, 192), (sk, hkv, 128)))
  o = A.attention(q, k, v, **kw)
  do = torch.randn_like(o)
  got = torch.autograd.grad(o, (q, k, v), do)
  qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
  w = ref.attention(qf, kf, vf, **kw)
  want = torch.autograd.grad(w, (qf, kf, vf), do.float())
  for name, g, r in zip("dq dk dv".split(), got, want):
    assert bool(torch.isfinite(g).all()), name
    assert ((g.float() - r).norm() / r.norm()).item() < bound, name


@pytest.mark.parametrize("b,s,hq,hkv", [(1, 63, 2, 2), (1, 64, 2, 1), (2, 65, 2, 2), (1, 128, 4, 4), (2, 129, 2, 1),
                                        (1, 300, 16, 16), (1, 1024, 2, 2)])
@pytest.mark.parametrize("causal", [True, False])
def test_lengths_and_groups(cuda_lib, b, s, hq, hkv, causal):
  _check(b, s, s, hq, hkv, causal=causal)


@pytest.mark.parametrize("sq,sk", [(100, 260), (64, 129), (257, 400)])
def test_more_keys_than_queries(cuda_lib, sq, sk):
  _check(1, sq, sk, 2, 2, causal=True)


@pytest.mark.parametrize("window", [40, 64, 100])
def test_window(cuda_lib, window):
  _check(1, 320, 320, 2, 1, causal=True, window=window)


@pytest.mark.parametrize("s", [129, 256, 321])
def test_segments(cuda_lib, s):
  g = torch.Generator(device="cuda").manual_seed(s)
  cuts = torch.randint(0, s, (2, 3), device="cuda", generator=g)
  ids = (torch.arange(s, device="cuda")[None, :, None] >= cuts[:, None, :]).sum(-1).to(torch.int32)
  _check(2, s, s, 2, 2, causal=True, q_segment_ids=ids)
  _check(2, s, s, 2, 2, causal=False, q_segment_ids=torch.randint(0, 3, (2, s), device="cuda", generator=g).to(torch.int32))


def test_positions(cuda_lib):
  pos = torch.cat([torch.arange(64, 128), torch.arange(256, 320)]).to("cuda", torch.int32)[None]
  _check(1, 128, 384, 2, 2, causal=True, q_positions=pos.long())


ROUNDED = 1.66e-3     # relative error (2-norm) of values rounded to bf16 once


@pytest.mark.parametrize("sq,sk,kind", [(77, 77, "plain"), (1024, 1024, "plain"), (300, 300, "full"), (77, 77, "segments"),
                                        (300, 300, "segments"), (1024, 1024, "segments"), (300, 300, "window"),
                                        (257, 400, "plain"), (128, 384, "positions")])
def test_roundings(cuda_lib, sq, sk, kind):
  """Against 64 bits.  Plain calls round P and dS to bf16 once each, the forward's result in delta and the gradient itself;
  masked ones and those with more keys than queries keep fp32 probabilities, so that only the gradient is rounded."""
  g = torch.Generator(device="cuda").manual_seed(sq)
  q, k, v, do = (torch.randn(2, s, 4, d, device="cuda", generator=g).to(torch.bfloat16)
                 for s, d in ((sq, 192), (sk, 192), (sk, 128), (sq, 128)))
  kw = {"causal": kind != "full"}
  if kind == "segments":
    cuts = torch.randint(0, sq, (2, 4), device="cuda", generator=g)
    kw["q_segment_ids"] = (torch.arange(sq, device="cuda")[None, :, None] >= cuts[:, None, :]).sum(-1).to(torch.int32)
  if kind == "window":
    kw["window"] = 100
  if kind == "positions":
    kw["q_positions"] = torch.cat([torch.arange(64, 128), torch.arange(256, 320)]).to("cuda")[None].expand(2, -1).contiguous()
  lead = [t.requires_grad_(True) for t in (q, k, v)]
  got = torch.autograd.grad(A.attention(*lead, **kw), lead, do)
  exact = [t.detach().double().requires_grad_(True) for t in lead]
  keep = ref.build_mask(sq, sk, "cuda", **kw)
  p = (torch.einsum("bqhd,bkhd->bhqk", exact[0], exact[1]) * 192 ** -0.5).masked_fill(~keep, float("-inf")).softmax(-1)
  want = torch.autograd.grad(torch.einsum("bhqk,bkhd->bqhd", p, exact[2]), exact, do.double())
  fine = kind in ("segments", "window", "positions") or sq != sk
  for name, a, w in zip("dq dk dv".split(), got, want):
    err = ((a.double() - w).norm() / w.norm()).item()
    assert err < (1.03 * ROUNDED if fine else 3 ** 0.5 * ROUNDED), (name, err)


def test_reproducible(cuda_lib):
  torch.manual_seed(0)
  q, k = (torch.randn(1, 700, 4, 192, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
  v = torch.randn(1, 700, 4, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  do = torch.randn(1, 700, 4, 128, device="cuda", dtype=torch.bfloat16)
  a = torch.autograd.grad(A.attention(q, k, v), (q, k, v), do)
  for _ in range(3):
    for x, y in zip(a, torch.autograd.grad(A.attention(q, k, v), (q, k, v), do)):
      assert torch.equal(x, y)
