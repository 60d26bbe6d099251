"""sm_100a flash attention (forward and backward) against the eager fp32 reference."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import reference as ref


def _rel(got, want):
  return ((got.float() - want.float()).norm() / (want.float().norm() + 1e-12)).item()


def _qkv(b, s, hq, hkv, d, dv=128, fused=True, seed=0):
  torch.manual_seed(seed)
  if fused and d == dv:
    buf = torch.randn(b, s, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16)
    q = buf[..., : hq * d].view(b, s, hq, d)
    k = buf[..., hq * d: (hq + hkv) * d].view(b, s, hkv, d)
    v = buf[..., (hq + hkv) * d:].view(b, s, hkv, d)
    return q, k, v
  q = torch.randn(b, s, hq, d, device="cuda", dtype=torch.bfloat16)
  k = torch.randn(b, s, hkv, d, device="cuda", dtype=torch.bfloat16)
  v = torch.randn(b, s, hkv, dv, device="cuda", dtype=torch.bfloat16)
  return q, k, v


FWD_CASES = [
  # b, s, hq, hkv, d, causal, window
  (1, 128, 1, 1, 128, True, None),
  (1, 256, 2, 1, 128, True, None),
  (2, 384, 4, 2, 128, True, None),
  (1, 200, 2, 2, 128, True, None),
  (1, 320, 2, 1, 128, False, None),
  (1, 1024, 4, 1, 128, True, None),
  (1, 512, 2, 1, 128, True, 100),
  (1, 256, 2, 2, 192, True, None),
  (2, 2048, 4, 2, 128, True, None),     # several batch rows at a length with many key blocks
  (1, 8192, 4, 1, 128, True, None),     # the training sequence length
]


@pytest.mark.parametrize("b,s,hq,hkv,d,causal,window", FWD_CASES)
def test_attention_forward(cuda_lib, b, s, hq, hkv, d, causal, window):
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(b, s, hq, hkv, d)
  o, lse = A.attn_fwd(q, k, v, causal=causal, window=window)
  want, want_lse = ref.attention(q, k, v, causal=causal, window=window, return_lse=True)
  torch.cuda.synchronize()
  assert _rel(o, want) < 2e-2, _rel(o, want)
  assert torch.allclose(lse, want_lse, atol=2e-2, rtol=1e-3), (lse - want_lse).abs().max()


def test_attention_forward_segments_and_positions(cuda_lib):
  from torchprime_b200.ops import attention_sm100 as A
  b, s, hq, hkv, d = 2, 256, 2, 1, 128
  q, k, v = _qkv(b, s, hq, hkv, d, seed=3)
  seg = torch.zeros(b, s, dtype=torch.int32, device="cuda")
  seg[0, 100:] = 1
  seg[1, 30:200] = 1
  seg[1, 200:] = 2
  o, _ = A.attn_fwd(q, k, v, causal=True, q_seg=seg.reshape(-1).contiguous(), kv_seg=seg.reshape(-1).contiguous())
  want = ref.attention(q, k, v, causal=True, q_segment_ids=seg)
  assert _rel(o, want) < 2e-2
  # rows of a zig-zag context-parallel shard: queries are chunks 0 and 3 of 4, keys are all 4 chunks
  pos = torch.cat([torch.arange(0, 64), torch.arange(192, 256)]).to(torch.int32).cuda()
  qs = q[:, pos.long()].contiguous()
  o2, _ = A.attn_fwd(qs, k, v, causal=True, q_pos=pos.repeat(b).contiguous())
  want2 = ref.attention(qs, k, v, causal=True, q_positions=pos.long())
  assert _rel(o2, want2) < 2e-2


BWD_CASES = [
  (1, 128, 1, 1, 128, True, None),
  (1, 256, 4, 1, 128, True, None),
  (2, 384, 4, 2, 128, True, None),
  (1, 200, 2, 2, 128, True, None),
  (1, 320, 2, 1, 128, False, None),
  (1, 512, 2, 1, 128, True, 100),
  (1, 256, 2, 2, 192, True, None),
  (2, 2048, 4, 2, 128, True, None),
  (1, 8192, 2, 1, 128, True, None),     # the training sequence length
]


@pytest.mark.parametrize("b,s,hq,hkv,d,causal,window", BWD_CASES)
def test_attention_backward(cuda_lib, b, s, hq, hkv, d, causal, window):
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(b, s, hq, hkv, d, fused=False, seed=5)
  do = torch.randn(b, s, hq, 128, device="cuda", dtype=torch.bfloat16)
  o, lse = A.attn_fwd(q, k, v, causal=causal, window=window)
  dq, dk, dv = A.attn_bwd(do, q, k, v, o, lse, causal=causal, window=window)
  qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
  ref.attention(qf, kf, vf, causal=causal, window=window).backward(do.float())
  torch.cuda.synchronize()
  assert _rel(dv, vf.grad) < 3e-2, ("dv", _rel(dv, vf.grad))
  assert _rel(dk, kf.grad) < 3e-2, ("dk", _rel(dk, kf.grad))
  assert _rel(dq, qf.grad) < 3e-2, ("dq", _rel(dq, qf.grad))


@pytest.mark.parametrize("s,window,segments", [(4096, None, 0), (4097, 300, 0), (4230, None, 9), (4230, 130, 9)])
def test_backward_lists_its_query_tiles(cuda_lib, s, window, segments):
  """Key blocks that see all, few and scattered query tiles, more than one warp counts at a time; bound of the cases above."""
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(1, s, 2, 1, 128, fused=False, seed=s)
  do = torch.randn(1, s, 2, 128, device="cuda", dtype=torch.bfloat16)
  ids = ((torch.arange(s, device="cuda") * segments // s) % 4).to(torch.int32)[None].contiguous() if segments else None
  o, lse = A.attn_fwd(q, k, v, causal=True, window=window, q_seg=ids, kv_seg=ids)
  got = A.attn_bwd(do, q, k, v, o, lse, causal=True, window=window, q_seg=ids, kv_seg=ids)
  leaves = [t.float().requires_grad_(True) for t in (q, k, v)]
  ref.attention(*leaves, causal=True, window=window, q_segment_ids=ids).backward(do.float())
  for g, w in zip(got, leaves):
    assert _rel(g, w.grad) < 2e-2, _rel(g, w.grad)


def test_backward_keeps_nan(cuda_lib):
  """A NaN in one query row reaches the gradients of every key that the row sees, also through the tiles without a mask."""
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(1, 640, 2, 1, 128, fused=False, seed=3)
  q[0, 600, 0, 7] = float("nan")
  do = torch.randn(1, 640, 2, 128, device="cuda", dtype=torch.bfloat16)
  o, lse = A.attn_fwd(q, k, v, causal=True)
  dq, dk, dv = A.attn_bwd(do, q, k, v, o, lse, causal=True)
  assert not torch.isfinite(dv[0, :601]).any() and not torch.isfinite(dk[0, :601]).any()
  assert not torch.isfinite(dq[0, 600, 0]).any()
  assert torch.isfinite(dv[0, 601:]).all() and torch.isfinite(dq[0, :600]).all() and torch.isfinite(dq[0, :, 1]).all()


def test_attention_autograd_fused_qkv(cuda_lib):
  from torchprime_b200.ops import functional as ops
  b, s, hq, hkv, d = 1, 256, 4, 2, 128
  torch.manual_seed(9)
  buf = torch.randn(b, s, (hq + 2 * hkv) * d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  q = buf[..., : hq * d].view(b, s, hq, d)
  k = buf[..., hq * d: (hq + hkv) * d].view(b, s, hkv, d)
  v = buf[..., (hq + hkv) * d:].view(b, s, hkv, d)
  o = ops.attention(q, k, v, causal=True)
  assert ops.attention_impl_in_use().startswith("sm100")
  do = torch.randn_like(o)
  o.backward(do)
  bf = buf.detach().float().requires_grad_(True)
  qf = bf[..., : hq * d].view(b, s, hq, d)
  kf = bf[..., hq * d: (hq + hkv) * d].view(b, s, hkv, d)
  vf = bf[..., (hq + hkv) * d:].view(b, s, hkv, d)
  ref.attention(qf, kf, vf, causal=True).backward(do.float())
  assert _rel(buf.grad, bf.grad) < 3e-2


@pytest.mark.parametrize("b,s,hq,hkv,causal,window,cap", [(1, 384, 4, 2, True, None, 2.0), (2, 300, 2, 1, True, 100, 5.0),
                                                          (1, 256, 2, 2, False, None, 1.0), (1, 1024, 4, 1, True, None, 30.0)])
def test_attention_logit_soft_cap(cuda_lib, b, s, hq, hkv, causal, window, cap):
  """Scores capped as cap * tanh(s / cap) inside the kernels, forward and backward (the reference's
  splash-attention option attn_logits_soft_cap, torchprime/utils/kernel_utils.py:30-37)."""
  from torchprime_b200.ops import attention_sm100 as A
  from torchprime_b200.ops import functional as ops
  q, k, v = _qkv(b, s, hq, hkv, 128, fused=False, seed=11)
  q = (q * 2).contiguous()       # scores well into the curved part of the cap
  do = torch.randn(b, s, hq, 128, device="cuda", dtype=torch.bfloat16)
  o, lse = A.attn_fwd(q, k, v, causal=causal, window=window, softcap=cap)
  want, want_lse = ref.attention(q, k, v, causal=causal, window=window, softcap=cap, return_lse=True)
  assert _rel(o, want) < 2e-2, _rel(o, want)
  assert torch.allclose(lse, want_lse, atol=2e-2, rtol=1e-3), (lse - want_lse).abs().max()
  dq, dk, dv = A.attn_bwd(do, q, k, v, o, lse, causal=causal, window=window, softcap=cap)
  qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
  ref.attention(qf, kf, vf, causal=causal, window=window, softcap=cap).backward(do.float())
  torch.cuda.synchronize()
  assert _rel(dv, vf.grad) < 3e-2, ("dv", _rel(dv, vf.grad))
  assert _rel(dk, kf.grad) < 3e-2, ("dk", _rel(dk, kf.grad))
  assert _rel(dq, qf.grad) < 3e-2, ("dq", _rel(dq, qf.grad))
  # the public op takes the kernel path too
  qa = q.clone().requires_grad_(True)
  oa = ops.attention(qa, k, v, causal=causal, window=window, softcap=cap)
  assert ops.attention_impl_in_use().startswith("sm100")
  oa.backward(do)
  assert _rel(qa.grad, qf.grad) < 3e-2


@pytest.mark.parametrize("dqk", [128, 192])
@pytest.mark.parametrize("sq,sk", [(300, 64), (513, 100), (200, 30)])
@pytest.mark.parametrize("window", [None, 350])
def test_forward_and_backward_with_more_queries_than_keys_and_no_causal_mask(cuda_lib, dqk, sq, sk, window):
  """Queries whose natural position lies before the first key see every key unless the mask is causal."""
  from torchprime_b200.ops import attention_sm100 as A
  torch.manual_seed(sq)
  q, k, v = (torch.randn(1, s, h, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
             for s, h, d in ((sq, 4, dqk), (sk, 2, dqk), (sk, 2, 128)))
  o = A.attention(q, k, v, causal=False, window=window)
  do = torch.randn_like(o)
  got = torch.autograd.grad(o, (q, k, v), do)
  qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
  w = ref.attention(qf, kf, vf, causal=False, window=window)
  want = torch.autograd.grad(w, (qf, kf, vf), do.float())
  for a, r in zip((o, *got), (w, *want)):
    assert ((a.float() - r.float()).norm() / r.float().norm()).item() < 2e-2


@pytest.mark.parametrize("dqk", [128, 192])
def test_forward_of_rows_without_keys(cuda_lib, dqk):
  """Rows that see no key (positions before the first one, an id that no key has) give zeros, next to rows that do."""
  from torchprime_b200.ops import attention_sm100 as A
  torch.manual_seed(0)
  q, k = (torch.randn(1, 200, 2, dqk, device="cuda", dtype=torch.bfloat16) for _ in range(2))
  v = torch.randn(1, 200, 2, 128, device="cuda", dtype=torch.bfloat16)
  pos = torch.arange(200, device="cuda")[None] - 37
  got = A.attention(q, k, v, causal=True, q_positions=pos)
  want = ref.attention(q.float(), k.float(), v.float(), causal=True, q_positions=pos)
  assert bool((got[:, :37] == 0).all()) and _rel(got[:, 37:], want[:, 37:]) < 2e-2
  ids = (torch.arange(200, device="cuda") % 3)[None].int()
  got = A.attention(q, k, v, causal=False, q_segment_ids=ids, kv_segment_ids=torch.zeros_like(ids))
  want = ref.attention(q.float(), k.float(), v.float(), causal=False, q_segment_ids=ids, kv_segment_ids=torch.zeros_like(ids))
  assert bool((got[:, ids[0] != 0] == 0).all()) and _rel(got[:, ids[0] == 0], want[:, ids[0] == 0]) < 2e-2


def test_backward_is_the_same_with_and_without_a_mask(cuda_lib):
  """Segment ids that are all one (256 keys: no table of ranges, so every tile is masked) change no bit of any gradient."""
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(2, 256, 4, 2, 128, fused=False, seed=11)
  q = (3 * q).to(torch.bfloat16)
  do = torch.randn(2, 256, 4, 128, device="cuda", dtype=torch.bfloat16)
  ids = torch.zeros(2, 256, device="cuda", dtype=torch.int32)
  o, lse = A.attn_fwd(q, k, v, causal=False)
  plain = A.attn_bwd(do, q, k, v, o, lse, causal=False)
  masked = A.attn_bwd(do, q, k, v, o, lse, causal=False, q_seg=ids, kv_seg=ids)
  assert all(torch.equal(a, b) for a, b in zip(plain, masked))


def test_backward_nan_is_nan_everywhere_it_reaches(cuda_lib):
  """Not an infinity, which a check for NaN lets through."""
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(1, 640, 2, 1, 128, fused=False, seed=3)
  q[0, 600, 0, 7] = float("nan")
  do = torch.randn(1, 640, 2, 128, device="cuda", dtype=torch.bfloat16)
  o, lse = A.attn_fwd(q, k, v, causal=True)
  dq, dk, dv = A.attn_bwd(do, q, k, v, o, lse, causal=True)
  assert torch.isnan(dv[0, :601]).all() and torch.isnan(dk[0, :601]).all() and torch.isnan(dq[0, 600, 0]).all()


def test_backward_rows_behind_the_last_add_nothing(cuda_lib):
  """A last tile of two queries holds the next sequence's gradients in its other rows; their probability is 0, whatever
  stands there (2^-126 of 1e37 would be seen)."""
  from torchprime_b200.ops import attention_sm100 as A
  q, _, _ = _qkv(2, 130, 2, 1, 128, fused=False, seed=5)
  _, k, v = _qkv(2, 128, 2, 1, 128, fused=False, seed=6)
  v = (1e-3 * v).to(torch.bfloat16)
  do = torch.randn(2, 130, 2, 128, device="cuda").to(torch.bfloat16)
  do[1] = 1e37
  o, lse = A.attn_fwd(q, k, v, causal=False)
  both = A.attn_bwd(do, q, k, v, o, lse, causal=False)
  o, lse = A.attn_fwd(q[:1], k[:1], v[:1], causal=False)
  one = A.attn_bwd(do[:1], q[:1], k[:1], v[:1], o, lse, causal=False)
  assert all(torch.equal(a[:1], b) for a, b in zip(both, one))


@pytest.mark.parametrize("b,s,hq,hkv,d", [(3, 300, 6, 3, 128), (1, 40000, 4, 2, 128), (5, 9000, 2, 1, 128), (1, 30000, 3, 3, 192)])
def test_forward_covers_every_tile_of_every_group_of_heads(cuda_lib, b, s, hq, hkv, d):
  """Heads in one group, in groups of one key head and in groups of which the last is smaller: rows of every head, first and
  last tile of each sequence among them, against fp32; the rest finite."""
  from torchprime_b200.ops import attention_sm100 as A
  q, k, v = _qkv(b, s, hq, hkv, d, fused=False, seed=s)
  o, lse = A.attn_fwd(q, k, v, causal=True)
  assert torch.isfinite(o).all() and torch.isfinite(lse).all()
  for i in range(b):
    for r in (0, 127, 128, s // 2, s - 129, s - 1):
      for h in range(hq):
        sc = (k[i, :r + 1, h * hkv // hq].float() @ q[i, r, h].float()) / d ** 0.5
        want = sc.softmax(0) @ v[i, :r + 1, h * hkv // hq].float()
        assert _rel(o[i, r, h], want) < 2e-2 and abs(lse[i, h, r].item() - sc.logsumexp(0).item()) < 1e-2
