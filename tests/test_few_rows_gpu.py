"""GEMMs with few rows (csrc/gemm_skinny_sm100.cu): dense and grouped by expert."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import kernels as k, moe
from torchprime_b200.ops._lib import lib, ptr, stream_ptr

BF16_EPS = 2.0 ** -8


def _skinny(x, w, *, a_mn=False, b_mn=False, epi=k.EPI_BF16, alpha=1.0, aux=None, w2=None, c2=None, nt=0, splits=0, out=None):
  t, kk = x.shape[::-1] if a_mn else x.shape
  n = w.shape[1] if b_mn else w.shape[0]
  n *= 2 if w2 is not None else 1
  n_out = n // 2 if epi == k.EPI_SWIGLU else n
  if out is None:
    out = torch.empty(t, n_out, device="cuda", dtype=torch.float32 if epi == k.EPI_F32 else torch.bfloat16)
  rc = lib().tpb_gemm_skinny_bf16(ptr(x), ptr(w), ptr(w2), ptr(out), t, n, kk, x.stride(0), w.stride(0), out.stride(0),
                                  int(a_mn), int(b_mn), epi, alpha, ptr(aux), aux.stride(0) if aux is not None else 0, ptr(c2),
                                  c2.stride(0) if c2 is not None else 0, nt, splits, stream_ptr())
  assert rc == 0, rc
  return out


@pytest.fixture(autouse=True)
def _signature():
  from ctypes import c_float as F, c_int as I, c_longlong as LL, c_void_p as P
  fn = lib().tpb_gemm_skinny_bf16
  fn.argtypes, fn.restype = [P, P, P, P, I, I, I, LL, LL, LL, I, I, I, F, P, LL, P, LL, I, I, P], I


def _close(got, want, scale):
  """One rounding to the result's type plus fp32 sums in another order (``scale``: size of the terms' sum)."""
  err = (got.float() - want).abs()
  eps = BF16_EPS if got.dtype == torch.bfloat16 else 0.0
  assert bool((err <= eps * want.abs() + 2e-6 * scale).all()), (err - eps * want.abs()).max()


@pytest.mark.parametrize("t,nt", [(1, 0), (15, 0), (16, 16), (17, 0), (33, 32), (64, 0), (77, 0), (128, 0), (129, 128), (50, 16)])
@pytest.mark.parametrize("n,kk,splits", [(8, 64, 1), (128, 72, 0), (136, 520, 2), (1000, 2048, 0), (264, 1096, 8), (384, 256, 4)])
def test_dense_layouts_and_epilogues(cuda_lib, t, nt, n, kk, splits):
  torch.manual_seed(t * 1000 + n)
  x = torch.randn(t, kk + 16, device="cuda", dtype=torch.bfloat16)[:, 8:kk + 8]       # rows with a pitch
  w = torch.randn(n, kk, device="cuda", dtype=torch.bfloat16)
  res = torch.randn(t, n + 8, device="cuda", dtype=torch.bfloat16)[:, :n]
  want = x.double() @ w.double().t()
  scale = float(kk)
  # results land in the middle of a larger buffer whose border must stay as it is
  for b_mn in (False, True):
    ww = w.t().contiguous() if b_mn else w
    for epi, aux, ref_ in ((k.EPI_BF16, None, want), (k.EPI_F32, None, want), (k.EPI_BF16_RES, res, want + res.double())):
      big = torch.full((t + 2, n + 16), 7.0, device="cuda", dtype=torch.float32 if epi == k.EPI_F32 else torch.bfloat16)
      out = big[1:t + 1, 8:n + 8]
      _skinny(x, ww, b_mn=b_mn, epi=epi, aux=aux, nt=nt, splits=splits, out=out)
      _close(out, ref_, scale)
      out.fill_(7.0)
      assert bool((big == 7.0).all())


@pytest.mark.parametrize("t", [33, 48, 49, 79, 80, 81, 97, 112, 113, 130, 200, 300])
@pytest.mark.parametrize("b_mn", [False, True])
def test_tiles_of_any_multiple_of_sixteen_rows(cuda_lib, t, b_mn):
  """Tiles narrower than the instantiation they run in, with every split of the contraction and a last tile that is not full."""
  torch.manual_seed(t)
  x, w = (torch.randn(r, 1160, device="cuda", dtype=torch.bfloat16) for r in (t, 200))
  want = x.double() @ w.double().t()
  ww = w.t().contiguous() if b_mn else w
  for splits in (0, 1, 2, 4, 8):
    _close(_skinny(x, ww, b_mn=b_mn, splits=splits), want, 1160.0)
  for nt in (48, 80, 96, 112):
    assert torch.equal(_skinny(x, ww, b_mn=b_mn, nt=nt, splits=4), _skinny(x, ww, b_mn=b_mn, nt=128, splits=4))


@pytest.mark.parametrize("t", [1, 16, 40, 128])
@pytest.mark.parametrize("f,kk,splits", [(8, 64, 1), (72, 136, 2), (192, 1024, 8), (1408, 512, 0)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_dense_swiglu(cuda_lib, t, f, kk, splits, b_mn):
  torch.manual_seed(f)
  x = torch.randn(t, kk, device="cuda", dtype=torch.bfloat16)
  g, u = (torch.randn(f, kk, device="cuda", dtype=torch.bfloat16) / kk ** 0.5 for _ in range(2))
  gate, up = x.double() @ g.double().t(), x.double() @ u.double().t()
  want = torch.nn.functional.silu(gate) * up
  both = torch.cat([g, u])
  lay = (lambda m: m.t().contiguous()) if b_mn else (lambda m: m)
  for w, w2 in ((lay(both), None), (lay(g), lay(u))):
    gu = torch.empty(t, 2 * f, device="cuda", dtype=torch.bfloat16)
    act = _skinny(x, w, b_mn=b_mn, epi=k.EPI_SWIGLU, w2=w2, c2=gu, splits=splits)
    _close(gu, torch.cat([gate, up], -1), 8.0)
    # silu amplifies an error of the gate by at most 1.1
    err = (act.double() - want).abs()
    assert bool((err <= BF16_EPS * want.abs() + 1e-5 * (1 + up.abs())).all()), err.max()


@pytest.mark.parametrize("m,n", [(8, 64), (64, 200), (72, 128), (136, 264), (576, 2048)])
@pytest.mark.parametrize("t,splits", [(1, 1), (63, 0), (64, 1), (200, 2), (1500, 8)])
def test_weight_gradient(cuda_lib, m, n, t, splits):
  """C = dY^T X: both operands contracted over their rows."""
  torch.manual_seed(m + t)
  dy = torch.randn(t, m, device="cuda", dtype=torch.bfloat16)
  x = torch.randn(t, n, device="cuda", dtype=torch.bfloat16)
  want = dy.double().t() @ x.double()
  for epi in (k.EPI_BF16, k.EPI_F32):
    for nt in (0, 64, 128):
      _close(_skinny(dy, x, a_mn=True, b_mn=True, epi=epi, nt=nt, splits=splits), want, float(max(t, 16)))


def test_split_sums_do_not_depend_on_the_run(cuda_lib):
  x = torch.randn(40, 4096, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(512, 4096, device="cuda", dtype=torch.bfloat16)
  a = _skinny(x, w, epi=k.EPI_F32, splits=8)
  for _ in range(3):
    assert torch.equal(a, _skinny(x, w, epi=k.EPI_F32, splits=8))


@pytest.mark.parametrize("align", [16, 32])
@pytest.mark.parametrize("t,kk,e", [(1, 6, 64), (4, 6, 64), (37, 2, 8), (128, 8, 256), (5, 1, 3)])
def test_plan_with_narrow_segments(cuda_lib, align, t, kk, e):
  torch.manual_seed(t)
  idx = torch.randint(0, e, (t, kk), device="cuda", dtype=torch.int32)      # repeated experts in a token too
  plan = moe._build_dispatch_plan_kernel(idx, e, align)
  assert plan.num_rows % align == 0 and int(plan.k_offsets[-1]) <= plan.num_rows
  flat = idx.reshape(-1).long()
  order = torch.argsort(flat, stable=True)
  counts = torch.bincount(flat, minlength=e)
  off = torch.cat([counts.new_zeros(1), ((counts + align - 1) // align * align).cumsum(0)])
  assert torch.equal(plan.k_offsets.long(), off) and torch.equal(plan.counts.long(), counts)
  rank = torch.arange(flat.numel(), device="cuda") - (counts.cumsum(0) - counts)[flat[order]]
  dest = torch.empty_like(flat)
  dest[order] = off[flat[order]] + rank
  assert torch.equal(plan.dest.reshape(-1).long(), dest)
  pair = torch.full((plan.num_rows,), -1, device="cuda")
  pair[dest] = torch.arange(flat.numel(), device="cuda")
  assert torch.equal(plan.src_pair, pair)
  assert torch.equal(plan.src_row.long(), torch.where(pair >= 0, pair // kk, pair))
  tiles = torch.arange(plan.num_rows // align, device="cuda") * align
  te = torch.bucketize(tiles, off[1:], right=True)
  assert torch.equal(plan.tile_expert.long(), torch.where(te < e, te, torch.full_like(te, -1)))


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("t,kk,e,d,f", [(1, 6, 64, 256, 192), (4, 6, 64, 2048, 1408), (16, 2, 8, 512, 1024), (190, 2, 16, 256, 320),
                                        (48, 1, 2, 128, 64), (260, 6, 64, 128, 64)])
def test_grouped_mlp_without_gradients(cuda_lib, t, kk, e, d, f, fused):
  """The few-rows path against the tiled grouped GEMMs' oracle, one expert hit by nobody."""
  torch.manual_seed(t + e)
  x = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
  wg, wu = ((torch.randn(e, d, f, device="cuda") / d ** 0.5).to(torch.bfloat16) for _ in range(2))
  wd = (torch.randn(e, f, d, device="cuda") / f ** 0.5).to(torch.bfloat16)
  if fused:
    wg = torch.cat([wg, wu], dim=2)
  logits = torch.randn(t, e, device="cuda")
  logits[:, 0] = -1e9
  w, idx, _ = moe.router_topk(logits, kk, mode="softmax")
  with torch.no_grad():
    y = moe.grouped_mlp(x, w, idx, wg, None if fused else wu, wd, fused_gate_up=fused)
  want = moe.grouped_mlp_reference(x.double(), w.double(), idx, wg.double(), wu.double(), wd.double(), fused)
  # act and rows are rounded to bf16 once each, the result once more
  assert ((y.double() - want).norm() / want.norm()).item() < 3 * BF16_EPS


@pytest.mark.parametrize("t,kk,e", [(40, 2, 8), (90, 1, 4), (33, 6, 64)])
def test_grouped_mlp_with_uneven_routing(cuda_lib, t, kk, e):
  """All tokens go to the same experts, which then span several segment steps; the other experts get nothing."""
  torch.manual_seed(t)
  d, f = 256, 128
  x = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
  wg, wu = ((torch.randn(e, d, f, device="cuda") / 16).to(torch.bfloat16) for _ in range(2))
  wd = (torch.randn(e, f, d, device="cuda") / 11).to(torch.bfloat16)
  idx = torch.arange(kk, device="cuda", dtype=torch.int32).flip(0)[None].expand(t, -1).contiguous()
  w = torch.rand(t, kk, device="cuda")
  align = moe.few_rows_align(t, kk, e)
  assert align is not None and t > align
  with torch.no_grad():
    y = moe.grouped_mlp(x, w, idx, wg, wu, wd)
  want = moe.grouped_mlp_reference(x.double(), w.double(), idx, wg.double(), wu.double(), wd.double())
  assert ((y.double() - want).norm() / want.norm()).item() < 3 * BF16_EPS


def test_route_of_the_few_rows_path():
  assert moe.few_rows_align(4, 6, 64) == 16 and moe.few_rows_align(128, 6, 64) == 16
  assert moe.few_rows_align(96, 2, 8) == 32 and moe.few_rows_align(97, 2, 8) is None
  assert moe.few_rows_align(256, 6, 64) == 32 and moe.few_rows_align(257, 6, 64) is None


def test_recomputed_forward_gives_the_recorded_bits(cuda_lib):
  """A forward that will be repeated with gradients runs the same kernels as the repetition."""
  from torchprime_b200.ops import functional as ops
  torch.manual_seed(0)
  t, kk, e, d, f = 40, 2, 8, 1024, 512
  assert moe.few_rows_align(t, kk, e) is not None
  x = torch.randn(t, d, device="cuda", dtype=torch.bfloat16)
  wg, wu = ((torch.randn(e, d, f, device="cuda") / 32).to(torch.bfloat16) for _ in range(2))
  wd = (torch.randn(e, f, d, device="cuda") / 32).to(torch.bfloat16).requires_grad_(True)
  w, idx, _ = moe.router_topk(torch.randn(t, e, device="cuda"), kk)
  recorded = moe.grouped_mlp(x, w, idx, wg, wu, wd)
  assert recorded.requires_grad
  with torch.no_grad(), ops.recomputed_forward():
    assert torch.equal(moe.grouped_mlp(x, w, idx, wg, wu, wd), recorded)


def test_no_tokens(cuda_lib):
  """Without tokens no expert is hit: an empty result, recorded or not."""
  assert moe.few_rows_align(0, 6, 64) is None
  wg, wu = (torch.randn(8, 128, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
  wd = torch.randn(8, 64, 128, device="cuda", dtype=torch.bfloat16)
  x = torch.empty(0, 128, device="cuda", dtype=torch.bfloat16)
  w, idx = torch.empty(0, 2, device="cuda"), torch.empty(0, 2, device="cuda", dtype=torch.int32)
  for recorded in (False, True):
    with torch.set_grad_enabled(recorded):
      y = moe.grouped_mlp(x, w, idx, wg, wu, wd)
    assert y.shape == (0, 128) and y.dtype == x.dtype


def test_linear_f32_logits(cuda_lib):
  from torchprime_b200.ops import functional as ops
  x = torch.randn(3, 256, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(1000, 256, device="cuda", dtype=torch.bfloat16)
  with torch.no_grad():
    got = ops.linear_f32(x, w)
  assert got.dtype == torch.float32
  _close(got, x.double() @ w.double().t(), 256.0)
  w.requires_grad_(True)
  assert ops.linear_f32(x, w).requires_grad


@pytest.mark.parametrize("shift", [0.0, 0.5])
@pytest.mark.parametrize("t,n,kk", [(1, 64, 2048), (4, 102400, 2048), (1500, 64, 2048), (16, 256, 7168), (17, 1000, 520), (33, 8, 8),
                                    (2, 136, 72), (300, 256, 7168)])
def test_linear_f32_is_as_exact_as_fp32(cuda_lib, t, n, kk, shift):
  """Distance from 64 bits: what an MMA gives for 16 products and the sum are cut to 24 bits once each (2^-24 of
  their size on average); and not above the fp32 library product's by more than the last rounding."""
  from torchprime_b200.ops import functional as ops
  torch.manual_seed(t + n)
  x = (torch.randn(t, kk, device="cuda") + shift).to(torch.bfloat16)
  w = ((torch.randn(n, kk, device="cuda") + shift) / 50).to(torch.bfloat16)
  want = torch.cat([x.double() @ part.double().t() for part in w.split(8192)], 1)
  far = lambda y: ((y.double() - want).norm() / want.norm()).item()  # noqa: E731
  with torch.no_grad():
    got = far(ops.linear_f32(x, w))
  assert got < 2.0 ** -23
  assert got < far(torch.nn.functional.linear(x.float(), w.float())) + 2.0 ** -25


def test_linear_f32_not_finite(cuda_lib):
  from torchprime_b200.ops import functional as ops
  x = torch.randn(20, 512, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(64, 512, device="cuda", dtype=torch.bfloat16)
  x[3, 7], x[4, 500], x[18, 0] = float("inf"), float("-inf"), float("nan")
  with torch.no_grad():
    got = ops.linear_f32(x, w)
  want = torch.nn.functional.linear(x.float(), w.float())
  assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[3:5], want[3:5])


@pytest.mark.parametrize("M,N,K", [(1, 64, 128), (77, 512, 256), (128, 1000, 136), (300, 512, 512), (700, 64, 2048),
                                   (32, 512, 64), (33, 512, 264), (64, 264, 512), (65, 264, 512), (128, 264, 1024), (129, 256, 1024),
                                   (1100, 1024, 1024), (1300, 1024, 1024), (900, 2048, 2048), (1200, 2048, 2048)])
def test_route_of_a_gemm_call(cuda_lib, M, N, K):
  """Calls the rule gives to this kernel against the tiled kernel (max_ctas keeps a call there)."""
  torch.manual_seed(M)
  x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) / K ** 0.5
  res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
  for b_mn in (False, True):
    ww = w.t().contiguous() if b_mn else w
    for epi, aux in ((k.EPI_BF16, None), (k.EPI_F32, None), (k.EPI_BF16_RES, res), (k.EPI_SWIGLU, None)):
      if epi == k.EPI_SWIGLU and (N // 2) % 8:
        continue
      a = k.gemm(x, ww, b_mn=b_mn, epi=epi, aux=aux, alpha=0.5)
      b = k.gemm(x, ww, b_mn=b_mn, epi=epi, aux=aux, alpha=0.5, max_ctas=148)
      # two fp32 sums of K random terms in other orders: each strays by about 2^-24 sqrt(K / 2) of the result
      bound = 2.0 ** -23 * K ** 0.5
      assert ((a.float() - b.float()).norm() / b.float().norm()).item() < (bound if epi == k.EPI_F32 else 2.0 ** -9)


@pytest.mark.parametrize("m,n,kk", [(512, 4096, 4096), (1024, 2048, 4096)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_fp32_results_that_a_split_tile_does_not_take_stay_here(cuda_lib, m, n, kk, b_mn):
  """Products that the rule of the split tiles names too, with an epilogue they do not have: this kernel's bits, which
  adds in another order than the tiled one."""
  g = torch.Generator("cuda").manual_seed(m)
  a = torch.randn(m, kk, device="cuda", generator=g).to(torch.bfloat16)
  b = torch.randn(*((kk, n) if b_mn else (n, kk)), device="cuda", generator=g).to(torch.bfloat16)
  want = _skinny(a, b, b_mn=b_mn, epi=k.EPI_F32)
  assert torch.equal(k.gemm(a, b, b_mn=b_mn, epi=k.EPI_F32), want)
  assert not torch.equal(k.gemm(a, b, b_mn=b_mn, epi=k.EPI_F32, max_ctas=148), want)      # (the tiled kernel)


@pytest.mark.parametrize("m,n,few_rows", [(9472, 256, True), (9472, 512, False)])      # 37 and 74 tiles of 256 x 256
def test_split_tiles_that_take_a_wave_more_are_not_taken(cuda_lib, m, n, few_rows):
  """One tile more than clusters of four fit the chip once, and twice: the kernels that do not split tiles by pairs."""
  kk = 8192
  g = torch.Generator("cuda").manual_seed(m)
  a = torch.randn(m, kk, device="cuda", generator=g).to(torch.bfloat16)
  b = torch.randn(n, kk, device="cuda", generator=g).to(torch.bfloat16)
  want = _skinny(a, b) if few_rows else k.gemm(a, b, max_ctas=148)
  assert torch.equal(k.gemm(a, b), want)


@pytest.mark.parametrize("shape", [(1, 1), (4, 1), (16, 1), (2, 17), (3, 32), (128, 1)])
@pytest.mark.parametrize("n1,n2,kk", [(3072, 576, 2048), (136, 128, 1024), (8, 264, 1096)])
def test_two_products_of_one_input(cuda_lib, shape, n1, n2, kk):
  """One launch for both against 64 bits; the projections' own launches give the same to the order of fp32 sums."""
  from torchprime_b200.ops import functional as ops
  torch.manual_seed(n1 + shape[0])
  x = torch.randn(*shape, kk, device="cuda", dtype=torch.bfloat16)
  w1, w2 = (torch.randn(n, kk, device="cuda", dtype=torch.bfloat16) for n in (n1, n2))
  with torch.no_grad():
    nat = ops._native().linear_pair(x, w1, w2)
    both = ops.linear_pair(x, w1, w2)
  rows = shape[0] * shape[1]
  assert (nat is not None) == (rows <= 32 or 8 * rows <= kk)
  for y, w in zip(both, (w1, w2)):
    assert y.shape == (*shape, w.shape[0])
    _close(y, x.double() @ w.double().t(), float(kk))
    if nat is None:
      assert torch.equal(y, ops.linear(x, w))


def test_two_products_refuse_what_one_launch_cannot_do(cuda_lib):
  """Other types, layouts and alignments, and calls with a graph, go through the ordinary projections."""
  from torchprime_b200.ops import functional as ops
  nat = ops._native()
  x = torch.randn(4, 1024, device="cuda", dtype=torch.bfloat16)
  w1, w2 = (torch.randn(n, 1024, device="cuda", dtype=torch.bfloat16) for n in (256, 128))
  buf = torch.randn(4 * 1024 + 8, device="cuda", dtype=torch.bfloat16)
  with torch.no_grad():
    assert nat.linear_pair(x, w1, w2) is not None
    for a, b, c in ((x.float(), w1, w2), (x, w1.t(), w2), (x, w1, w2[:, :512]), (x[:0], w1, w2), (buf[1:4097].view(4, 1024), w1, w2),
                    (x, w1[:255], w2), (torch.randn(200, 1024, device="cuda").bfloat16(), w1, torch.randn(40000, 1024, device="cuda").bfloat16())):
      assert nat.linear_pair(a, b, c) is None
  assert nat.linear_pair(x, w1, w2) is None
  w1.requires_grad_(True)
  y1, y2 = ops.linear_pair(x, w1, w2)
  assert y1.requires_grad and not y2.requires_grad


@pytest.mark.parametrize("rows", [900, 2100])
def test_two_products_allocate_nothing_where_they_do_not_run(cuda_lib, rows):
  from torchprime_b200.ops import functional as ops
  x = torch.randn(rows, 1024, device="cuda", dtype=torch.bfloat16)
  w1, w2 = (torch.randn(n, 1024, device="cuda", dtype=torch.bfloat16) for n in (3072, 576))
  before = torch.cuda.memory_stats()["allocation.all.allocated"]
  with torch.no_grad():
    assert ops._native().linear_pair(x, w1, w2) is None
  assert torch.cuda.memory_stats()["allocation.all.allocated"] == before


@pytest.mark.parametrize("rows", [129, 200, 300, 469])
@pytest.mark.parametrize("n1,n2,kk", [(3072, 576, 2048), (1536, 576, 5120), (1024, 264, 1032)])
def test_two_products_of_more_rows_than_a_tile(cuda_lib, rows, n1, n2, kk):
  """Several token tiles, the second product's behind the first one's in the grid."""
  from torchprime_b200.ops import functional as ops
  torch.manual_seed(rows)
  x = torch.randn(rows, kk, device="cuda", dtype=torch.bfloat16)
  w1, w2 = (torch.randn(n, kk, device="cuda", dtype=torch.bfloat16) for n in (n1, n2))
  with torch.no_grad():
    both = ops.linear_pair(x, w1, w2)
  for y, w in zip(both, (w1, w2)):
    _close(y, x.double() @ w.double().t(), float(kk))
