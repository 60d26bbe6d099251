"""Attention kernels skip key blocks that share no segment with a query tile (ranges of the ids)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import attention_sm100 as A
from torchprime_b200.ops import reference as ref
from torchprime_b200.ops._lib import check, lib, ptr, stream_ptr


def _ids(kind, b, s):
  g = torch.Generator(device="cuda").manual_seed(s + b)
  if kind == "sorted":
    cuts = torch.randint(0, s, (b, 5), device="cuda", generator=g)
    at = torch.arange(s, device="cuda")
    return (at[None, :, None] >= cuts[:, None, :]).sum(-1).to(torch.int32)
  if kind == "one":
    return torch.full((b, s), 3, dtype=torch.int32, device="cuda")
  if kind == "blocks":       # ids that change at tile edges, decreasing, with the int32 extremes
    at = torch.arange(s, device="cuda") // 64
    ids = (-at).to(torch.int32)
    ids[at == 0] = 2 ** 31 - 1
    ids[at == at.max()] = -2 ** 31
    return ids.expand(b, s).contiguous()
  return torch.randint(-2, 2, (b, s), device="cuda", generator=g).to(torch.int32)   # no order at all


@pytest.mark.parametrize("s", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("kind", ["sorted", "blocks", "mixed"])
def test_range_tables(cuda_lib, s, kind):
  ids = _ids(kind, 3, s)
  n = (s + 63) // 64
  out = torch.empty(3, n, 2, dtype=torch.int32, device="cuda")
  check(lib().tpb_attn_seg_ranges(ptr(ids), ptr(out), 3, s, stream_ptr()), "seg_ranges")
  for i in range(n):
    part = ids[:, 64 * i:64 * (i + 1)]
    assert torch.equal(out[:, i, 0], part.amin(-1)) and torch.equal(out[:, i, 1], part.amax(-1))


@pytest.mark.parametrize("causal,window", [(True, None), (False, None), (True, 70)])
@pytest.mark.parametrize("s", [40, 129, 256, 257, 320, 777])
@pytest.mark.parametrize("kind", ["sorted", "one", "blocks", "mixed"])
def test_forward_and_backward(cuda_lib, s, kind, causal, window):
  """Against the fp32 definition; the bound is that of the unsegmented kernels' tests."""
  torch.manual_seed(s)
  b, hq, hkv = 2, 4, 2
  q, k, v = (torch.randn(b, s, h, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (hq, hkv, hkv))
  ids = _ids(kind, b, s)
  o = A.attention(q, k, v, causal=causal, window=window, q_segment_ids=ids)
  do = torch.randn_like(o)
  got = torch.autograd.grad(o, (q, k, v), do)
  qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
  w = ref.attention(qf, kf, vf, causal=causal, window=window, q_segment_ids=ids)
  want = torch.autograd.grad(w, (qf, kf, vf), do.float())
  for g, r in zip((o, *got), (w, *want)):
    assert ((g.float() - r.float()).norm() / r.float().norm()).item() < 2e-2


def test_keys_and_queries_with_other_ids(cuda_lib):
  """Key ids of their own: a query tile whose segment no key has gives zeros and zero gradients."""
  q, k, v = (torch.randn(1, 400, 2, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
  q_seg = torch.zeros(1, 400, dtype=torch.int32, device="cuda")
  kv_seg = torch.zeros(1, 400, dtype=torch.int32, device="cuda")
  q_seg[:, 128:256] = 9
  o = A.attention(q, k, v, causal=False, q_segment_ids=q_seg, kv_segment_ids=kv_seg)
  dq, dk, dv = torch.autograd.grad(o, (q, k, v), torch.randn_like(o))
  assert bool((o[:, 128:256] == 0).all()) and bool((dq[:, 128:256] == 0).all())
  assert bool(torch.isfinite(dk).all()) and bool(torch.isfinite(dv).all()) and bool((dv != 0).any())


@pytest.mark.parametrize("s,window", [(63, 2), (65, 64), (130, 65), (200, 127), (300, None)])
@pytest.mark.parametrize("positions", ["natural", "reversed halves"])
def test_masks_as_bits(cuda_lib, s, window, positions):
  """Masks of 64-score words: window edges inside and at the words' ends, explicit positions, many segments in a warp."""
  torch.manual_seed(s)
  q, k, v = (torch.randn(2, s, h, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (4, 2, 2))
  ids = torch.randint(0, 40, (2, s), device="cuda").sort(dim=-1)[0].to(torch.int32)
  ids[1] = torch.randint(0, 3, (s,), device="cuda")
  pos, q_ids = None, ids
  if positions != "natural":
    pos = torch.cat([torch.arange(s // 2, s), torch.arange(0, s // 2)]).to("cuda", torch.int32).expand(2, s).contiguous()
    q_ids = ids.gather(1, pos.long())     # (a query sees at least the key at its own position)
  o = A.attention(q, k, v, causal=True, window=window, q_segment_ids=q_ids, kv_segment_ids=ids, q_positions=pos)
  do = torch.randn_like(o)
  got = torch.autograd.grad(o, (q, k, v), do)
  qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
  w = ref.attention(qf, kf, vf, causal=True, window=window, q_segment_ids=q_ids, kv_segment_ids=ids,
                    q_positions=None if pos is None else pos.long())
  want = torch.autograd.grad(w, (qf, kf, vf), do.float())
  for g, r in zip((o, *got), (w, *want)):
    assert torch.isfinite(g).all()
    assert ((g.float() - r.float()).norm() / r.float().norm()).item() < 2e-2


def _both(q, k, v, **kw):
  leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
  o = A.attention(*leaves, **kw)
  o.backward(torch.linspace(-1, 1, o.numel(), device="cuda").view(o.shape).to(o.dtype))
  return [o.detach()] + [t.grad for t in leaves]


@pytest.mark.parametrize("sq,sk", [(70, 70), (300, 300), (200, 70)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("window", [2 ** 31 - 1, 2 ** 31 - 66, 2 ** 30 + 1])
def test_a_window_wider_than_any_sequence_is_none(cuda_lib, sq, sk, causal, window):
  """No sum of a position and the window wraps (more queries than keys: positions before the first key)."""
  g = torch.Generator(device="cuda").manual_seed(sq + sk)
  q, k, v = (torch.randn(2, s, 2, 128, device="cuda", generator=g).to(torch.bfloat16) for s in (sq, sk, sk))
  for got, want in zip(_both(q, k, v, causal=causal, window=window), _both(q, k, v, causal=causal)):
    assert torch.equal(got, want)


@pytest.mark.parametrize("first", [2 ** 30 - 3, 2 ** 30 + 100])
def test_positions_far_past_the_last_key_see_all_of_them(cuda_lib, first):
  g = torch.Generator(device="cuda").manual_seed(first % 1000)
  q, k, v = (torch.randn(2, 150, 2, 128, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
  pos = (first + torch.arange(300, device="cuda", dtype=torch.int32) % 150).view(2, 150)
  for got, want in zip(_both(q, k, v, causal=True, q_positions=pos), _both(q, k, v, causal=False)):
    assert torch.equal(got, want)
