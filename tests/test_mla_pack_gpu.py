"""Key / value layout passes of latent attention."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import functional as ops


@pytest.mark.parametrize("b,s,heads,dn,dr,dv", [(1, 1, 1, 8, 8, 8), (2, 37, 16, 128, 64, 128), (1, 5, 3, 24, 16, 40),
                                                (1, 300, 128, 128, 64, 128)])
def test_mla_pack(cuda_lib, b, s, heads, dn, dr, dv):
  torch.manual_seed(s)
  kv = torch.randn(b, s, heads * (dn + dv), device="cuda", dtype=torch.bfloat16, requires_grad=True)
  rot = torch.randn(b, s, dr, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  kk, v = ops.mla_pack(kv, rot, heads, dn, dv)
  kv4 = kv.view(b, s, heads, dn + dv)
  assert torch.equal(v, kv4[..., dn:]) and kk.is_contiguous() and v.is_contiguous()
  assert torch.equal(kk, torch.cat([kv4[..., :dn], rot[:, :, None].expand(b, s, heads, dr)], -1))
  dk, dv_ = torch.randn_like(kk), torch.randn_like(v)
  dkv, drot = torch.autograd.grad([kk, v], [kv, rot], [dk, dv_])
  assert torch.equal(dkv.view_as(kv4), torch.cat([dk[..., :dn], dv_], -1))
  want = dk[..., dn:].double().sum(2)
  assert bool(((drot.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * heads * 4).all())


# Heads that leave a group of four or a round of thirty-two partly filled, more vectors to a row than a warp has lanes, and
# more tokens than one pass of the grid takes.
@pytest.mark.parametrize("b,s,heads,dn,dr,dv", [(2, 9, 5, 264, 512, 8), (1, 17, 33, 8, 24, 272), (1, 3, 70, 16, 256, 16),
                                                (1, 20001, 2, 8, 16, 8), (1, 524300, 1, 8, 8, 8)])
def test_mla_pack_edges(cuda_lib, b, s, heads, dn, dr, dv):
  test_mla_pack(cuda_lib, b, s, heads, dn, dr, dv)


@pytest.mark.parametrize("b,s,at", [(1, 1, 0), (1, 130, 3), (3, 37, 5), (2, 8, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_mla_pack_into_a_cache(cuda_lib, b, s, at, dtype):
  heads, dn, dr, dv, room = 5, 24, 16, 40, 160
  kv = torch.randn(b, s, heads * (dn + dv), device="cuda", dtype=torch.bfloat16)
  rot = torch.randn(b, s, dr, device="cuda", dtype=torch.bfloat16)
  kc = torch.full((b + 1, room, heads, dn + dr), 7.0, device="cuda", dtype=dtype)
  vc = torch.full((b + 1, room, heads, dv), 7.0, device="cuda", dtype=dtype)
  want_k, want_v = kc.clone(), vc.clone()
  want_k[:b, at:at + s], want_v[:b, at:at + s] = ops.mla_pack(kv, rot, heads, dn, dv)
  ops.mla_pack_into(kv, rot, heads, dn, dv, kc[:b, at:at + s], vc[:b, at:at + s])
  assert torch.equal(kc, want_k) and torch.equal(vc, want_v)


def test_latent_split(cuda_lib):
  x = torch.randn(2, 9, 48, device="cuda", dtype=torch.bfloat16, requires_grad=True)
  a, b = ops.latent_split(x, 32)
  assert torch.equal(torch.cat([a, b], -1), x)
  (g,) = torch.autograd.grad([a, b], [x], [torch.ones_like(a), 2 * torch.ones_like(b)])
  assert bool((g[..., :32] == 1).all()) and bool((g[..., 32:] == 2).all())
  (g,) = torch.autograd.grad(ops.latent_split(x, 32)[1].sum(), x)
  assert bool((g[..., :32] == 0).all()) and bool((g[..., 32:] == 1).all())
