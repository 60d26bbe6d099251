"""The tiled GEMM's results leave through shared memory and TMA: edges of C and what lies around it."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import kernels as k, moe


@pytest.mark.parametrize("M", [129, 160, 200, 257, 700])
@pytest.mark.parametrize("N", [8, 40, 64, 104, 264, 520])
@pytest.mark.parametrize("epi", [k.EPI_BF16, k.EPI_F32, k.EPI_F32_ACC])
def test_nothing_around_the_result_is_written(cuda_lib, M, N, epi):
  torch.manual_seed(M + N)
  a = torch.randn(M, 136, device="cuda", dtype=torch.bfloat16)
  b = torch.randn(N, 136, device="cuda", dtype=torch.bfloat16)
  dt = torch.bfloat16 if epi == k.EPI_BF16 else torch.float32
  big = torch.full((M + 2, N + 16), 5.0, device="cuda", dtype=dt)
  out = big[1:M + 1, 8:N + 8]
  start = torch.randn(M, N, device="cuda") if epi == k.EPI_F32_ACC else torch.zeros(M, N, device="cuda")
  out.copy_(start)
  k.gemm(a, b, out=out, epi=epi)
  want = a.double() @ b.double().t() + start.double()
  err = (out.double() - want).abs()
  assert bool((err <= (2.0 ** -8 if dt == torch.bfloat16 else 0.0) * want.abs() + 2e-6 * 136).all()), err.max()
  out.fill_(5.0)
  assert bool((big == 5.0).all())


@pytest.mark.parametrize("M,F", [(130, 8), (200, 72), (300, 136), (513, 320)])
def test_swiglu_halves_do_not_run_into_each_other(cuda_lib, M, F):
  torch.manual_seed(F)
  a = torch.randn(M, 128, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(2 * F, 128, device="cuda", dtype=torch.bfloat16) / 11
  gu = torch.full((M + 1, 2 * F), 5.0, device="cuda", dtype=torch.bfloat16)
  act = k.gemm(a, w, epi=k.EPI_SWIGLU, c2=gu[:M])
  want = a.double() @ w.double().t()
  assert bool(((gu[:M].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all())
  ref_act = torch.nn.functional.silu(want[:, :F]) * want[:, F:]
  assert bool(((act.double() - ref_act).abs() <= 2.0 ** -8 * ref_act.abs() + 2e-4 * (1 + want[:, F:].abs())).all())
  assert bool((gu[M] == 5.0).all())


@pytest.mark.parametrize("da,db,dtype", [(72, 40, torch.bfloat16), (256, 136, torch.float32), (320, 512, torch.bfloat16)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_per_expert_weight_gradients(cuda_lib, da, db, dtype, accumulate):
  """Experts with few rows, one with none (zeros, or what was there)."""
  torch.manual_seed(da)
  e = 5
  idx = torch.randint(0, e - 1, (190, 2), device="cuda", dtype=torch.int32)
  plan = moe.build_dispatch_plan(idx, e)
  m = plan.num_rows
  live = (plan.src_row >= 0)[:, None]
  a, b = (torch.randn(m, d, device="cuda", dtype=torch.bfloat16) * live for d in (da, db))
  out = torch.randn(e, da, db, device="cuda").to(dtype)
  before = out.double()
  moe.grouped_gemm_wgrad(a, b, plan, out, accumulate)
  off = plan.k_offsets.tolist()
  for x in range(e):
    want = a[off[x]:off[x + 1]].double().t() @ b[off[x]:off[x + 1]].double() + (before[x] if accumulate else 0.0)
    err = (out[x].double() - want).abs()
    assert bool((err <= (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs() + 1e-4).all()), (x, err.max())


@pytest.mark.parametrize("M", [20, 100, 300])
@pytest.mark.parametrize("N", [100, 101, 259])
@pytest.mark.parametrize("epi", [k.EPI_BF16, k.EPI_F32, k.EPI_F32_ACC])
def test_columns_that_end_inside_a_vector(cuda_lib, M, N, epi):
  """Rows of C with a 16-byte pitch but any number of columns: the rest of the row stays as it is."""
  torch.manual_seed(M + N)
  a = torch.randn(M, 136, device="cuda", dtype=torch.bfloat16)
  b = torch.randn(N, 136, device="cuda", dtype=torch.bfloat16)
  dt = torch.bfloat16 if epi == k.EPI_BF16 else torch.float32
  big = torch.full((M, (N + 15) // 8 * 8), 5.0, device="cuda", dtype=dt)
  out = big[:, :N]
  k.gemm(a, b, out=out, epi=epi)
  want = a.double() @ b.double().t() + (5.0 if epi == k.EPI_F32_ACC else 0.0)
  err = (out.double() - want).abs()
  assert bool((err <= (2.0 ** -8 if dt == torch.bfloat16 else 0.0) * want.abs() + 2e-6 * 136).all()), err.max()
  assert bool((big[:, N:] == 5.0).all())


@pytest.mark.parametrize("counts", [[1, 63, 64, 65], [128, 0, 129, 300]])
@pytest.mark.parametrize("align", [128, 256])
def test_weight_gradients_stop_at_the_padding(cuda_lib, counts, align):
  """An expert's contraction ends at the multiple of 64 behind its rows: what the rest of its segment holds is not read."""
  torch.manual_seed(align)
  idx = torch.cat([torch.full((c,), i) for i, c in enumerate(counts)])[:, None].to("cuda", torch.int32)
  plan = moe.build_dispatch_plan(idx, len(counts), row_align=align)
  a, b = (torch.randn(plan.num_rows, d, device="cuda", dtype=torch.bfloat16) for d in (72, 136))
  off = plan.k_offsets.tolist()
  out = torch.empty(len(counts), 72, 136, device="cuda", dtype=torch.float32)
  for x, c in enumerate(counts):
    for t in (a, b):
      t[off[x] + c:off[x + 1]] = 0.0
      t[off[x] + (c + 63) // 64 * 64:off[x + 1]] = float("nan")
  moe.grouped_gemm_wgrad(a, b, plan, out, False)
  for x, c in enumerate(counts):
    want = a[off[x]:off[x] + c].double().t() @ b[off[x]:off[x] + c].double()
    assert bool(((out[x].double() - want).abs() <= 2e-6 * max(c, 1) + 1e-6).all())


@pytest.mark.parametrize("m,n,kk", [(129, 8, 72), (255, 264, 520), (257, 1000, 64), (300, 136, 1000), (640, 512, 200)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_few_tiles_on_pairs_are_those_of_single_ctas(cuda_lib, m, n, kk, a_mn, b_mn):
  """Products of a few 256 x 256 tiles run on CTA pairs; the kernel for one CTA (a limit on CTAs asks for it) sums in the
  same order."""
  torch.manual_seed(m + n)
  m8 = (m + 7) // 8 * 8 if a_mn else m
  a = torch.randn(*((kk, m8) if a_mn else (m8, kk)), device="cuda").bfloat16()
  b = torch.randn(*((kk, n) if b_mn else (n, kk)), device="cuda").bfloat16()
  res = torch.randn(m8, n, device="cuda").bfloat16()
  for epi, aux in ((k.EPI_BF16, None), (k.EPI_F32, None), (k.EPI_BF16_RES, res)):
    got = k.gemm(a, b, a_mn=a_mn, b_mn=b_mn, epi=epi, aux=aux)
    assert torch.equal(got, k.gemm(a, b, a_mn=a_mn, b_mn=b_mn, epi=epi, aux=aux, max_ctas=148))
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    want = want + res.double() if aux is not None else want
    assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8
  if not a_mn and n % 16 == 0:
    assert torch.equal(k.gemm(a, b, b_mn=b_mn, epi=k.EPI_SWIGLU), k.gemm(a, b, b_mn=b_mn, epi=k.EPI_SWIGLU, max_ctas=148))
