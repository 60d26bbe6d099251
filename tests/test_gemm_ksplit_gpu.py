"""Two CTA pairs to a tile, each contracting over half of K (csrc/gemm_sm100.cu, KSPLIT)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import _lib, kernels as k


def _split(a, b, out, b_mn, aux=None):
  m, kk = a.shape
  n = b.shape[1] if b_mn else b.shape[0]
  rc = _lib.lib().tpb_gemm_ksplit_bf16(
    a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, kk, a.stride(0), b.stride(0), out.stride(0), 0, int(b_mn),
    k.EPI_BF16 if aux is None else k.EPI_BF16_RES, 1.0, None if aux is None else aux.data_ptr(),
    0 if aux is None else aux.stride(0), None, 0, _lib.stream_ptr())
  _lib.check(rc, "gemm_ksplit")


def _inputs(m, n, kk, b_mn, seed=0):
  g = torch.Generator("cuda").manual_seed(seed + m + n + kk)
  a = torch.randn(m, kk, device="cuda", generator=g).to(torch.bfloat16)
  b = torch.randn(*((kk, n) if b_mn else (n, kk)), device="cuda", generator=g).to(torch.bfloat16)
  return a, b, a.double() @ (b.double() if b_mn else b.double().t())


# K of two and three k-blocks and not a multiple of one; columns that end inside a tile, a half and a 64-wide box;
# more tiles than clusters are resident (the ring is used again after an exchange)
@pytest.mark.parametrize("m,n,kk", [(1, 8, 72), (129, 136, 128), (256, 264, 192), (300, 392, 1000), (513, 520, 2048),
                                    (2304, 2816, 136)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_result_and_what_lies_around_it(cuda_lib, m, n, kk, b_mn, residual):
  a, b, want = _inputs(m, n, kk, b_mn)
  big = torch.full((m + 2, n + 16), 5.0, device="cuda", dtype=torch.bfloat16)
  out = big[1:m + 1, 8:n + 8]
  aux = torch.randn(m, n, device="cuda").to(torch.bfloat16) if residual else None
  _split(a, b, out, b_mn, aux)
  if residual:
    want = want + aux.double()
  # bf16 rounding of the result, fp32 sums of kk products of N(0, 1) pairs
  assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-6 * kk).all())
  out.fill_(5.0)
  assert bool((big == 5.0).all())


def test_the_same_every_run(cuda_lib):
  a, b, _ = _inputs(512, 4096, 4096, False)
  outs = [torch.empty(512, 4096, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
  for o in outs:
    _split(a, b, o, False)
  assert all(torch.equal(o, outs[0]) for o in outs[1:])


def test_what_it_refuses(cuda_lib):
  a, b, _ = _inputs(256, 256, 64, False)          # one k-block
  with pytest.raises(_lib.KernelError):
    _split(a, b, torch.empty(256, 256, device="cuda", dtype=torch.bfloat16), False)
  a, b, _ = _inputs(256, 256, 128, False)
  with pytest.raises(_lib.KernelError):           # a residual that is not 16-byte aligned
    _split(a, b, torch.empty(256, 256, device="cuda", dtype=torch.bfloat16), False,
           aux=torch.empty(256 * 256 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(256, 256))


@pytest.mark.parametrize("m,n,kk", [(512, 4096, 4096), (1500, 4096, 8192), (900, 2048, 10944), (300, 6144, 4096)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_products_the_rule_gives_it(cuda_lib, m, n, kk, b_mn):
  """Through the general entry, with every epilogue (those it does not take go to the other kernels)."""
  a, b, want = _inputs(m, n, kk, b_mn)
  aux = torch.randn(m, n, device="cuda").to(torch.bfloat16)
  s = torch.tensor(0.5, device="cuda")
  tol = lambda w: 2.0 ** -8 * w.abs() + 2e-6 * kk      # noqa: E731
  for got, w in ((k.gemm(a, b, b_mn=b_mn), want), (k.gemm(a, b, b_mn=b_mn, epi=k.EPI_BF16_RES, aux=aux), want + aux.double()),
                 (k.gemm(a, b, b_mn=b_mn, scale=s), want / 2), (k.gemm(a, b, b_mn=b_mn, epi=k.EPI_F32), want)):
    assert bool(((got.double() - w).abs() <= tol(w)).all())
