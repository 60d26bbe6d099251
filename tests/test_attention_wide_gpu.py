"""Attention backward for query / key head dim 192 and value dim 128 against the fp32 definition."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import attention_sm100 as A
from torchprime_b200.ops import reference as ref

ROUNDED = 1.66e-3     # relative error (2-norm) of values rounded to bf16 once


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


def _ids(kind, b, s):
  g = torch.Generator(device="cuda").manual_seed(s + b)
  at = torch.arange(s, device="cuda")
  if kind == "sorted":
    cuts = torch.randint(0, s, (b, 5), device="cuda", generator=g)
    return (at[None, :, None] >= cuts[:, None, :]).sum(-1).to(torch.int32)
  if kind == "one":
    return torch.full((b, s), 3, dtype=torch.int32, device="cuda")
  if kind == "blocks":       # ids that change at tile edges, decreasing, with the int32 extremes
    ids = (-(at // 64)).to(torch.int32)
    ids[at < 64] = 2 ** 31 - 1
    ids[at // 64 == (s - 1) // 64] = -2 ** 31
    return ids.expand(b, s).contiguous()
  return torch.randint(-2, 2, (b, s), device="cuda", generator=g).to(torch.int32)   # no order at all


@pytest.mark.parametrize("causal,window", [(True, None), (False, None), (True, 70)])
@pytest.mark.parametrize("s", [257, 320, 777])
@pytest.mark.parametrize("kind", ["sorted", "one", "blocks", "mixed"])
def test_range_tables(cuda_lib, s, kind, causal, window):
  """Lengths with range tables: forward and gradients against the fp32 definition."""
  torch.manual_seed(s)
  q, k, v = (torch.randn(2, s, h, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
             for h, d in ((4, 192), (2, 192), (2, 128)))
  kw = {"causal": causal, "window": window, "q_segment_ids": _ids(kind, 2, s)}
  assert A._seg_ranges(kw["q_segment_ids"], kw["q_segment_ids"], 2, s, s)[0] is not None
  o = A.attention(q, k, v, **kw)
  do = torch.randn_like(o)
  got = torch.autograd.grad(o, (q, k, v), do)
  qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
  w = ref.attention(qf, kf, vf, **kw)
  want = torch.autograd.grad(w, (qf, kf, vf), do.float())
  # P is rounded once in the forward, o once; the gradients keep fp32 probabilities and are rounded once
  for a, r, bound in zip((o, *got), (w, *want), (2 ** 0.5, 1.1, 1.1, 1.1)):
    assert ((a.float() - r.float()).norm() / r.float().norm()).item() < bound * ROUNDED * 1.05


def test_keys_and_queries_with_other_ids(cuda_lib):
  """A query tile whose segment no key has, and a key block whose segment no query has, give zeros."""
  torch.manual_seed(0)
  q, k = (torch.randn(1, 400, 2, 192, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
  v = torch.randn(1, 400, 2, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  q_seg, kv_seg = (torch.zeros(1, 400, dtype=torch.int32, device="cuda") for _ in range(2))
  q_seg[:, 128:256] = 9
  kv_seg[:, 256:384] = 5
  o = A.attention(q, k, v, causal=False, q_segment_ids=q_seg, kv_segment_ids=kv_seg)
  dq, dk, dv = torch.autograd.grad(o, (q, k, v), torch.randn_like(o))
  for zero in (o[:, 128:256], dq[:, 128:256], dk[:, 256:384], dv[:, 256:384]):
    assert bool((zero == 0).all())
  for t in (o, dq, dk, dv):
    assert bool(torch.isfinite(t).all()) and bool((t[:, :128] != 0).any())


@pytest.mark.parametrize("kw", [{"causal": True}, {"causal": False}, {"causal": True, "window": 40}])
def test_more_queries_than_the_table_holds(cuda_lib, monkeypatch, kw):
  """The route of calls beyond the query-tile table, at a size that can be run."""
  monkeypatch.setattr(A, "_MAX_WIDE_QUERIES", 64)
  _check(2, 100, 100, 2, 2, **kw)
  ids = (torch.arange(100, device="cuda") // 30).to(torch.int32).expand(2, 100).contiguous()
  _check(2, 100, 100, 2, 2, q_segment_ids=ids, **kw)


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
