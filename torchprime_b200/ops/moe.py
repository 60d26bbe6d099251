"""Mixture-of-experts operators: routing, dropless (or capacity-limited) dispatch into an
expert-grouped row layout, grouped SwiGLU MLP, weighted combine.

What the reference does with argsort / one-hot / Pallas ``gmm`` calls
(torchprime/torch_xla_models/model/mixtral/model.py:302-626,
model/deepseek_v3/model.py:274-338) is organised here around one layout: the ``T*K``
(token, slot) pairs are sorted by expert and every expert's rows are padded to a multiple of
128, so a 128-row GEMM tile never straddles two experts and padded rows are zero.  All index
bookkeeping stays on the device (no host synchronisation): the padded row count is bounded
by ``T*K + 127*min(T*K, E)`` and tiles past the real end are marked unused.

On CUDA/bf16 the heavy parts run as sm_100a kernels (router top-k, row gather, grouped
tcgen05 GEMMs with fused SwiGLU, combine); elsewhere the same math runs in plain PyTorch.
"""

from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p
from dataclasses import dataclass

import torch
import torch.nn.functional as F

from . import _debug, _lib, reference as ref
from ._lib import check, lib, ptr, stream_ptr

P, I, LL, FL = c_void_p, c_int, c_longlong, c_float
_lib.register_signature("tpb_grouped_gemm_bf16", [P, P, P, P, I, I, I, I, LL, LL, LL, LL, I, I, I, FL, P, LL, I, P, P,
                                                  LL, I, P])
_lib.register_signature("tpb_grouped_wgrad_bf16", [P, P, P, I, I, I, I, LL, LL, LL, I, P, P, LL, P])
_lib.register_signature("tpb_router_topk", [P, I, P, P, P, P, I, I, I, I, I, I, I, FL, P])
_lib.register_signature("tpb_router_bwd", [P, I, P, P, P, P, I, I, I, I, I, FL, P])
_lib.register_signature("tpb_moe_plan", [P, I, I, I, I, I, P, P, P, P, P, P, P])
_lib.register_signature("tpb_moe_gather", [P, P, P, P, LL, I, P])
_lib.register_signature("tpb_moe_gather_real", [P, P, P, LL, I, P])
_lib.register_signature("tpb_grouped_gemm_skinny_bf16", [P, P, P, P, I, I, I, I, LL, LL, LL, LL, I, I, P, I, I, P])
_lib.register_signature("tpb_moe_combine", [P, P, P, P, LL, I, I, P])
_lib.register_signature("tpb_moe_combine_dw", [P, P, P, P, LL, I, I, P])

ROW_ALIGN = 128


def _kernels_ok(*ts) -> bool:
  from .functional import use_kernels
  return use_kernels(*ts)


# ----------------------------------------------------------------------------- routing
def _router_forward(lg, bias, k, mode, n_group, topk_group, norm_topk, scale):
  t, e = lg.shape
  w = torch.empty(t, k, dtype=torch.float32, device=lg.device)
  idx = torch.empty(t, k, dtype=torch.int32, device=lg.device)
  scores = torch.empty(t, e, dtype=torch.float32, device=lg.device)
  b = None
  if bias is not None:
    b = (bias if bias.dtype == torch.bfloat16 else bias.float()).contiguous()
  bf16 = int(lg.dtype == torch.bfloat16) + 2 * int(b is not None and b.dtype == torch.bfloat16)
  check(lib().tpb_router_topk(ptr(lg), bf16, ptr(b), ptr(w), ptr(idx), ptr(scores), t, e,
                              k, mode, n_group, topk_group, int(norm_topk), float(scale), stream_ptr()),
        "router_topk")
  return w, idx, scores


def _router_backward(lg, idx, dw, dscores, mode, norm_topk, scale):
  """The gradient of the logits in torch operators (for batched gradients)."""
  s = torch.softmax(lg.float(), dim=-1) if mode == 0 else torch.sigmoid(lg.float())
  ds = dscores if dscores is not None else torch.zeros_like(s)
  if dw is not None:
    sel, dsel = s.gather(1, idx.long()), dw * scale
    if norm_topk:
      total = sel.sum(-1, keepdim=True) + (0.0 if mode == 0 else 1e-20)
      dsel = (dsel - (dsel * sel).sum(-1, keepdim=True) / total) / total
    ds = ds + torch.zeros_like(s).scatter(1, idx.long(), dsel)
  g = s * (ds - (s * ds).sum(-1, keepdim=True)) if mode == 0 else ds * s * (1 - s)
  return g.to(lg.dtype)


class _RouterFn(torch.autograd.Function):
  """Kernels both ways; the backward re-derives the scores from the logits."""

  @staticmethod
  def forward(ctx, logits, bias, k, mode, n_group, topk_group, norm_topk, scale):
    lg = logits.contiguous()
    w, idx, scores = _router_forward(lg, bias, k, mode, n_group, topk_group, norm_topk, scale)
    ctx.save_for_backward(lg, idx)
    ctx.set_materialize_grads(False)
    ctx.args = (mode, norm_topk, scale)
    ctx.mark_non_differentiable(idx)
    return w, idx, scores

  @staticmethod
  def backward(ctx, dw, _didx, dscores):
    lg, idx = ctx.saved_tensors
    mode, norm_topk, scale = ctx.args
    if dw is None and dscores is None:
      return (None,) * 8
    from .functional import batched
    if batched(dw, dscores):
      return _router_backward(lg, idx, dw, dscores, mode, norm_topk, scale), None, None, None, None, None, None, None
    t, e = lg.shape
    dw = dw.float().contiguous() if dw is not None else None
    dscores = dscores.float().contiguous() if dscores is not None else None
    g = torch.empty_like(lg)
    check(lib().tpb_router_bwd(ptr(lg), int(lg.dtype == torch.bfloat16), ptr(idx), ptr(dw), ptr(dscores), ptr(g), t, e,
                               idx.shape[1], mode, int(norm_topk), float(scale), stream_ptr()), "router_bwd")
    return g, None, None, None, None, None, None, None


def router_topk(logits, k, mode="softmax", bias=None, n_group=1, topk_group=1, norm_topk=True, scale=1.0):
  """Returns (weights [T,K] fp32, indices [T,K] int32, scores [T,E] fp32).

  ``mode="softmax"``: Mixtral (softmax, top-k, renormalise).  ``mode="sigmoid"``: DeepSeek-V3
  (sigmoid, optional selection bias, group-limited top-k, normalise, scale)."""
  from .functional import _native
  m = 0 if mode == "softmax" else 1
  if (nat := _native()) is not None:
    r = nat.router_topk(logits, bias, k, m, n_group, topk_group, norm_topk, scale)
    if r is not None:
      return r
  e = logits.shape[-1]
  if logits.is_cuda and _kernels_ok() and e <= 256 and logits.dtype in (torch.float32, torch.bfloat16):
    return _RouterFn.apply(logits, bias, k, m, n_group, topk_group, norm_topk, scale)
  if m == 0:
    w, idx, s = ref.router_softmax_topk(logits, k, renormalize=norm_topk)
    return w * scale, idx.to(torch.int32), s
  w, idx, s = ref.router_sigmoid_group_topk(logits, bias, k, n_group, topk_group, norm_topk, scale)
  return w, idx.to(torch.int32), s


# ----------------------------------------------------------------------------- dispatch plan
@dataclass
class DispatchPlan:
  src_row: torch.Tensor      # [M] int32: token feeding padded row r, -1 for padding
  src_pair: torch.Tensor     # [M] int64: flat (token*K+slot) feeding row r, -1 for padding
  dest: torch.Tensor         # [T,K] int32: padded row of each pair, -1 if dropped
  tile_expert: torch.Tensor  # [M / min(row_align, 128)] int32
  k_offsets: torch.Tensor    # [E+1] int32 (multiples of row_align)
  counts: torch.Tensor       # [E] rows per expert (after dropping)
  num_rows: int              # M (static upper bound)
  num_experts: int
  top_k: int
  row_align: int = 128       # expert segments are padded to this many rows (256 lets the CTA-pair GEMM run;
                             # below 128 only grouped_mlp_few_rows can read the plan)


def pair_tiles_pay(per: float, experts: int) -> bool:
  """Whether segments of 256 rows, which let the grouped GEMMs use 256 x 256 CTA-pair tiles, are worth their padding for
  ``per`` rows per expert on average: a row costs 0.88 of what it does on 128-row tiles, so they are where the second half of the
  last segment is used by most experts, and from some segments on.  How many rows each expert gets is only known on the
  device; with many experts some are far from the average, and loads that differ take the first of the two away.  Time with 128-row
  segments over that with 256-row ones of the routed MLP, both passes; even loads / loads that differ by half an average / by a whole one:
      rows   8 experts, 4096 x 14336   16, 5120 x 8192       64, 2048 x 1408       128, 2048 x 768       256, 7168 x 2048
      100    1.03 / 1.11 / 1.08        0.93 / 0.93 / 0.97    0.92 / 0.98 / 0.95    0.85 / 0.90 / 0.94    0.91 / 0.94 / 0.97
      128    1.09 / 1.09 / 0.92        1.08 / 1.00 / 0.94    0.99 / 1.01 / 0.96    0.95 / 0.94 / 0.97    1.01 / 0.97 / 0.98
      144    1.18 / 1.19 / 1.02        1.15 / 0.99 / 0.98    1.10 / 0.99 / 0.97    1.08 / 0.96 / 0.94    1.16 / 0.95 / 0.97
      200    1.13 / 1.11 / 1.10        1.15 / 1.04 / 1.02    1.10 / 1.00 / 0.95    1.05 / 0.96 / 0.95    1.11 / 0.98 / 0.98
      240    1.15 / 1.01 / 0.98        1.13 / 1.02 / 1.03    1.12 / 1.01 / 0.96    1.06 / 1.00 / 0.98    1.10 / 1.02 / 0.97
      280    0.98 / 0.98 / 0.99        0.96 / 0.99 / 0.99    0.96 / 1.03 / 1.03    0.95 / 1.00 / 0.97    0.90 / 0.99 / 1.02
      352    1.04 / 1.17 / 1.10        1.02 / 1.08 / 1.03    0.98 / 1.09 / 1.03    0.96 / 0.99 / 0.99    0.92 / 0.99 / 0.99
      448    1.13 / 1.13 / 1.00        1.12 / 1.04 / 0.98    1.13 / 1.04 / 1.01    1.15 / 1.04 / 1.01    1.13 / 1.01 / 1.01
      600    1.01 / 1.07 / 1.03        0.95 / 1.06 / 1.04    1.04 / 1.06 / 1.03    1.03 / 1.05 / 1.05    0.95 / 0.99 / 1.01
      900    1.12 / 1.14 / 1.02        1.11 / 1.07 / 1.05    1.08 / 1.04 / 1.06    1.07 / 1.09 / 1.07    1.03 / 1.00 / 0.99
  The buffers hold the worst case, 127 or 255 rows more than its pairs for every expert: half as much again at 136 rows on average,
  another reason why many experts keep to 128 there."""
  if 528 <= per <= 640:
    return False
  if experts <= 16:
    return 128 <= per <= 240 or per >= 352
  return (experts <= 64 and 136 <= per <= 240) or per >= 448


def build_dispatch_plan(idx: torch.Tensor, num_experts: int, capacity: int | None = None,
                        rows_per_group: int | None = None, use_kernel: bool | None = None,
                        row_align: int | None = None) -> DispatchPlan:
  """Sort (token, slot) pairs by expert into 128-aligned segments, entirely on the device.

  ``capacity``: maximum rows per expert *per group of ``rows_per_group`` consecutive tokens*
  (the reference's "dropping" mode limits each expert per batch row); pairs beyond it are
  dropped (``dest = -1``)."""
  t, k = idx.shape
  e = num_experts
  dev = idx.device
  if row_align is None:
    row_align = 256 if capacity is None and pair_tiles_pay(t * k / e, e) else ROW_ALIGN
  assert row_align in (128, 256)
  if use_kernel is None:
    use_kernel = capacity is None and idx.is_cuda and _kernels_ok() and e <= 256
  if use_kernel:
    return _build_dispatch_plan_kernel(idx, e, row_align)
  align = row_align
  flat = idx.reshape(-1).long()
  n = flat.numel()
  if capacity is not None:
    grp = (torch.arange(n, device=dev) // k) // (rows_per_group or t)
    key = grp * e + flat
    order_g = torch.argsort(key, stable=True)
    sk = key[order_g]
    first = torch.ones(n, dtype=torch.bool, device=dev)
    first[1:] = sk[1:] != sk[:-1]
    start = torch.where(first, torch.arange(n, device=dev), torch.zeros((), dtype=torch.long, device=dev))
    start = torch.cummax(start, 0)[0]
    rank_g = torch.empty(n, dtype=torch.long, device=dev)
    rank_g[order_g] = torch.arange(n, device=dev) - start
    flat = torch.where(rank_g < capacity, flat, torch.full_like(flat, e))   # dropped pairs go to a sentinel
  order = torch.argsort(flat, stable=True)
  sorted_e = flat[order]
  # (torch.bincount reads the largest value back to the host; a scatter-add of ones does not)
  counts_all = torch.zeros(e + 1, dtype=torch.long, device=dev).scatter_add_(0, flat, torch.ones_like(flat))
  counts = counts_all[:e]
  padded = (counts + align - 1) // align * align
  ends_pad = torch.cumsum(padded, 0)
  off_pad = ends_pad - padded
  off = torch.cumsum(counts_all, 0) - counts_all
  rank = torch.arange(n, device=dev) - off[sorted_e]
  valid = sorted_e < e
  dest_sorted = torch.where(valid, torch.cat([off_pad, off_pad.new_zeros(1)])[sorted_e] + rank,
                            torch.full_like(rank, -1))
  # at most min(n, e) experts are hit (one segment step at least: without tokens gradients are still written)
  m = max(align, (n + (align - 1) * min(n, e) + align - 1) // align * align)
  dest = torch.empty(n, dtype=torch.long, device=dev)
  dest[order] = dest_sorted
  src_pair = torch.full((m + 1,), -1, dtype=torch.long, device=dev)
  src_pair[torch.where(valid, dest_sorted, torch.full_like(dest_sorted, m))] = order
  src_pair = src_pair[:m]
  src_row = torch.where(src_pair >= 0, src_pair // k, src_pair).to(torch.int32)
  tile_start = torch.arange(m // ROW_ALIGN, device=dev) * ROW_ALIGN
  te = torch.bucketize(tile_start, ends_pad, right=True)
  tile_expert = torch.where(te < e, te, torch.full_like(te, -1)).to(torch.int32)
  k_offsets = torch.cat([ends_pad.new_zeros(1), ends_pad]).to(torch.int32)
  return DispatchPlan(src_row=src_row.contiguous(), src_pair=src_pair, dest=dest.view(t, k).to(torch.int32).contiguous(),
                      tile_expert=tile_expert.contiguous(), k_offsets=k_offsets.contiguous(), counts=counts, num_rows=m,
                      num_experts=e, top_k=k, row_align=align)


def _build_dispatch_plan_kernel(idx: torch.Tensor, e: int, align: int = ROW_ALIGN) -> DispatchPlan:
  """The same plan from one kernel launch (a stable counting sort in one CTA or, from 1536 pairs on, in a cluster of eight)
  instead of about twenty-five torch kernels; nothing is read back to the host."""
  t, k = idx.shape
  dev = idx.device
  n = t * k
  # at most min(n, e) experts are hit (one segment step at least: without tokens gradients are still written)
  m = max(align, (n + (align - 1) * min(n, e) + align - 1) // align * align)
  tile = min(align, ROW_ALIGN)
  idx32 = idx.to(torch.int32).contiguous()
  ints = torch.empty(e + (e + 1) + n + m + m // tile, dtype=torch.int32, device=dev)
  counts, k_offsets, dest, src_row, tile_expert = torch.split(ints, [e, e + 1, n, m, m // tile])
  src_pair = torch.empty(m, dtype=torch.int64, device=dev)
  check(lib().tpb_moe_plan(ptr(idx32), t, k, e, m, align, ptr(counts), ptr(k_offsets), ptr(dest), ptr(src_row), ptr(src_pair),
                           ptr(tile_expert), stream_ptr()), "moe_plan")
  return DispatchPlan(src_row=src_row, src_pair=src_pair, dest=dest.view(t, k), tile_expert=tile_expert,
                      k_offsets=k_offsets, counts=counts, num_rows=m, num_experts=e, top_k=k, row_align=align)


# ----------------------------------------------------------------------------- raw kernels
def gather_rows(x, src_row, row_scale=None, pad=True):
  """``pad=False``: rows of index -1 are left unwritten (for readers that ignore them; no ``row_scale`` then)."""
  m, d = src_row.numel(), x.shape[-1]
  out = torch.empty(m, d, dtype=x.dtype, device=x.device)
  _debug.check_index("moe_gather", "src_row", src_row, 0, x.reshape(-1, d).shape[0], also_allowed=-1)
  if pad:
    check(lib().tpb_moe_gather(ptr(x), ptr(src_row), ptr(row_scale), ptr(out), m, d, stream_ptr()), "moe_gather")
  else:
    assert row_scale is None
    check(lib().tpb_moe_gather_real(ptr(x), ptr(src_row), ptr(out), m, d, stream_ptr()), "moe_gather_real")
  return out


def few_rows_align(t: int, k: int, e: int) -> int | None:
  """Token-tile width of the few-rows path for ``t`` tokens, or None where the tiled grouped GEMMs are as good.
  Both paths are bound by the weights of the experts that are hit; what counts is the average number of rows per
  expert (us for the routed MLP, tiled / 16 / 32 rows per segment step): 64 experts of 2048 x 1408, 6 rows 225 / 210 / 224,
  12 rows 228 / 217 / 226, 24 rows 231 / 268 / 231, 36 rows 234 / 337 / 286; 8 experts of 4096 x 14336, 8 rows 469 / 448 / 453,
  16 rows 471 / 485 / 454, 24 rows 555 / 525 / 459.  Without tokens no expert is hit and there is nothing for that path to
  launch."""
  per = t * k / e
  if per == 0:
    return None
  return 16 if per <= 12 else 32 if per <= 24 else None


def grouped_mlp_few_rows(x, weights, idx, w_gate, w_up, w_down, fused_gate_up, align):
  """The routed MLP without gradients when experts see a handful of rows each (decode): segments are
  padded to ``align`` rows instead of 128 and both GEMMs stream every hit expert's weights once."""
  t, k = idx.shape
  e, d = w_gate.shape[0], x.shape[1]
  f = w_down.shape[1]
  plan = _build_dispatch_plan_kernel(idx, e, align)
  m, hit = plan.num_rows, min(e, t * k)
  xg = gather_rows(x, plan.src_row, pad=False)
  act = torch.empty(m, f, dtype=x.dtype, device=x.device)
  rows = torch.empty(m, d, dtype=x.dtype, device=x.device)
  check(lib().tpb_grouped_gemm_skinny_bf16(
    ptr(xg), ptr(w_gate), None if fused_gate_up else ptr(w_up), ptr(act), m, 2 * f, d, e, d, w_gate.stride(1),
    w_gate.stride(0), f, 1, _lib.EPI_SWIGLU, ptr(plan.tile_expert), hit, align, stream_ptr()), "grouped_gemm_skinny gate/up")
  check(lib().tpb_grouped_gemm_skinny_bf16(
    ptr(act), ptr(w_down), None, ptr(rows), m, d, f, e, f, d, w_down.stride(0), d, 1, _lib.EPI_BF16,
    ptr(plan.tile_expert), hit, align, stream_ptr()), "grouped_gemm_skinny down")
  return combine_rows(rows, plan.dest, weights)


def combine_rows(rows, dest, w=None):
  t, k = dest.shape
  out = torch.empty(t, rows.shape[-1], dtype=rows.dtype, device=rows.device)
  _debug.check_index("moe_combine", "dest", dest, 0, rows.shape[0], also_allowed=-1)
  check(lib().tpb_moe_combine(ptr(rows), ptr(dest), ptr(w), ptr(out), t, k, rows.shape[-1], stream_ptr()),
        "moe_combine")
  return out


def combine_dw(rows, dest, dout):
  t, k = dest.shape
  dw = torch.empty(t, k, dtype=torch.float32, device=rows.device)
  _debug.check_index("moe_combine_dw", "dest", dest, 0, rows.shape[0], also_allowed=-1)
  check(lib().tpb_moe_combine_dw(ptr(rows), ptr(dest), ptr(dout), ptr(dw), t, k, rows.shape[-1], stream_ptr()),
        "moe_combine_dw")
  return dw


def grouped_gemm_rows(a, b, plan: DispatchPlan, *, b_mn: bool, b2=None, epi=_lib.EPI_BF16, out=None, c2=None,
                      n_total=None):
  """out[rows of e] = a[rows of e] @ B[e]^T.  ``b``: [E, N, K] (``b_mn=False``) or [E, K, N]
  (``b_mn=True``).  With ``epi=EPI_SWIGLU``: ``b`` = gate, ``b2`` = up (or ``b`` holds both
  halves along N when ``b2`` is None).  With ``epi=EPI_SWIGLU_BWD``: ``c2`` = [gate | up] before the activation,
  and the result is their gradient.  With other epilogues ``b2`` continues ``b`` along K: ``a`` then has 2K columns."""
  m, k = a.shape
  e = b.shape[0]
  n_one = b.shape[2] if b_mn else b.shape[1]
  swiglu = epi == _lib.EPI_SWIGLU
  n = n_total if n_total is not None else (2 * n_one if (swiglu and b2 is not None) else n_one)
  n_out = n // 2 if swiglu else 2 * n if epi == _lib.EPI_SWIGLU_BWD else n
  if out is None:
    out = torch.empty(m, n_out, dtype=torch.bfloat16, device=a.device)
  assert epi != _lib.EPI_SWIGLU_BWD or (c2 is not None and c2.shape == (m, n_out) and c2.stride(1) == 1)
  assert a.stride(1) == 1 and b.is_contiguous() and (b2 is None or b2.is_contiguous())
  ldb = b.stride(1)
  rc = lib().tpb_grouped_gemm_bf16(ptr(a), ptr(b), ptr(b2), ptr(out), m, n, k, e, a.stride(0), ldb, b.stride(0),
                                   out.stride(0), 0, int(b_mn), epi, 1.0, ptr(c2), c2.stride(0) if c2 is not None else 0,
                                   1, ptr(plan.tile_expert), None, 0, int(getattr(plan, "row_align", ROW_ALIGN)),
                                   stream_ptr())
  check(rc, f"grouped_gemm rows M={m} N={n} K={k} E={e}")
  return out


def grouped_dgrad_gate_up(dgu, w_gate, w_up, plan: DispatchPlan):
  """d_xg = dgu[:, :F] @ Wg[e]^T + dgu[:, F:] @ Wu[e]^T as one contraction over 2F (one fp32 sum, one
  rounding, no second pass over d_xg)."""
  f = w_gate.shape[2]
  if f % 64 == 0 and dgu.is_contiguous():
    return grouped_gemm_rows(dgu, w_gate, plan, b_mn=False, b2=w_up)
  d_xg = grouped_gemm_rows(dgu[:, :f], w_gate, plan, b_mn=False)
  return grouped_gemm_rows(dgu[:, f:], w_up, plan, b_mn=False, epi=_lib.EPI_BF16_ACC, out=d_xg)


def grouped_gemm_wgrad(a_rows, b_rows, plan: DispatchPlan, out, accumulate: bool):
  """out[e] (+)= a_rows[rows of e]^T @ b_rows[rows of e];  out: [E, Da, Db] bf16 or fp32."""
  e, da, db = out.shape
  assert a_rows.shape[1] == da and b_rows.shape[1] == db and out.is_contiguous()
  if out.dtype == torch.float32:
    epi = _lib.EPI_F32_ACC if accumulate else _lib.EPI_F32
  else:
    epi = _lib.EPI_BF16_ACC if accumulate else _lib.EPI_BF16
  # (the kernel's plan has its rows in front of each segment's padding, which then need not be read)
  counts = plan.counts if isinstance(plan, DispatchPlan) and plan.counts.dtype == torch.int32 else None
  rc = lib().tpb_grouped_wgrad_bf16(ptr(a_rows), ptr(b_rows), ptr(out), da, db, a_rows.shape[0], e, a_rows.stride(0),
                                    b_rows.stride(0), out.stride(1), epi, ptr(plan.k_offsets), ptr(counts), out.stride(0),
                                    stream_ptr())
  check(rc, f"grouped_gemm wgrad E={e} {da}x{db}")
  return out


# ----------------------------------------------------------------------------- grouped SwiGLU MLP
def _deliver_wgrad(w, compute):
  """Run ``compute(out, accumulate)`` into ``w.main_grad`` when present, else return a fresh gradient."""
  mg = getattr(w, "main_grad", None)
  if mg is not None:
    from .functional import overwrites_grad
    compute(mg, not overwrites_grad(w))
    w.grad_overwrite = False
    return None
  g = torch.empty(w.shape, dtype=torch.bfloat16, device=w.device)
  compute(g, False)
  return g


class _GroupedMLPFn(torch.autograd.Function):
  """y[t] = sum_k w[t,k] * down_e( silu(x[t] Wg_e) * (x[t] Wu_e) ),  e = idx[t,k]."""

  @staticmethod
  def forward(ctx, x, weights, w_gate, w_up, w_down, plan, fused_gate_up):
    xg = gather_rows(x, plan.src_row)
    need_grad = any(ctx.needs_input_grad)
    n2 = w_gate.shape[2] if fused_gate_up else 2 * w_gate.shape[2]
    gu = torch.empty(plan.num_rows, n2, dtype=x.dtype, device=x.device) if need_grad else None
    act = grouped_gemm_rows(xg, w_gate, plan, b_mn=True, b2=None if fused_gate_up else w_up, epi=_lib.EPI_SWIGLU, c2=gu,
                            n_total=n2)
    rows = grouped_gemm_rows(act, w_down, plan, b_mn=True)
    y = combine_rows(rows, plan.dest, weights)
    ctx.plan, ctx.fused = plan, fused_gate_up
    if need_grad:
      ctx.save_for_backward(x, weights, w_gate, w_up, w_down, xg, gu, act, rows)
    return y

  @staticmethod
  def backward(ctx, dy):
    x, weights, w_gate, w_up, w_down, xg, gu, act, rows = ctx.saved_tensors
    plan, fused = ctx.plan, ctx.fused
    dy = dy.contiguous()
    f = gu.shape[1] // 2
    dweights = combine_dw(rows, plan.dest, dy) if ctx.needs_input_grad[1] else None
    flat_w = torch.cat([weights.reshape(-1).float(), weights.new_zeros(1, dtype=torch.float32)])
    row_scale = flat_w[plan.src_pair].contiguous()          # -1 (padding) picks the appended zero
    d_rows = gather_rows(dy, plan.src_row, row_scale)
    # down projection: rows = act @ Wd[e]  (Wd [E, F, D])
    dgu = grouped_gemm_rows(d_rows, w_down, plan, b_mn=False, epi=_lib.EPI_SWIGLU_BWD, c2=gu)
    g_down = _deliver_wgrad(w_down, lambda out, acc: grouped_gemm_wgrad(act, d_rows, plan, out, acc))
    if fused:
      d_xg = grouped_gemm_rows(dgu, w_gate, plan, b_mn=False)
      g_gate = _deliver_wgrad(w_gate, lambda out, acc: grouped_gemm_wgrad(xg, dgu, plan, out, acc))
      g_up = None
    else:
      dg, du = dgu[:, :f], dgu[:, f:]
      d_xg = grouped_dgrad_gate_up(dgu, w_gate, w_up, plan)
      g_gate = _deliver_wgrad(w_gate, lambda out, acc: grouped_gemm_wgrad(xg, dg, plan, out, acc))
      g_up = _deliver_wgrad(w_up, lambda out, acc: grouped_gemm_wgrad(xg, du, plan, out, acc))
    dx = combine_rows(d_xg, plan.dest, None) if ctx.needs_input_grad[0] else None
    return dx, dweights, g_gate, g_up, g_down, None, None


def grouped_mlp_reference(x, weights, idx, w_gate, w_up, w_down, fused_gate_up=False, dropped=None):
  """Plain PyTorch: loop over experts (the oracle and the CPU path)."""
  t, k = idx.shape
  y = torch.zeros_like(x, dtype=torch.float32)
  e = w_gate.shape[0]
  for ex in range(e):
    sel = idx == ex
    if dropped is not None:
      sel = sel & ~dropped
    tok, slot = torch.nonzero(sel, as_tuple=True)
    if tok.numel() == 0:
      continue
    xi = x[tok]
    if fused_gate_up:
      gu = xi @ w_gate[ex]
      f = gu.shape[-1] // 2
      h = F.silu(gu[:, :f]) * gu[:, f:]
    else:
      h = F.silu(xi @ w_gate[ex]) * (xi @ w_up[ex])
    out = (h @ w_down[ex]).float() * weights[tok, slot].float()[:, None]
    y.index_add_(0, tok, out)
  return y.to(x.dtype)


def grouped_mlp(x, weights, idx, w_gate, w_up, w_down, *, fused_gate_up=False, capacity=None, rows_per_group=None):
  """Routed SwiGLU experts.  x [T,D]; weights/idx [T,K]; w_gate/w_up [E,D,F]; w_down [E,F,D]
  (``fused_gate_up``: w_gate is [E,D,2F] = [gate | up] and w_up is ignored).

  Calls without gradients and with a handful of rows per expert take :func:`grouped_mlp_few_rows`, whose sums are split
  differently; a forward that a backward pass will repeat says so with ``functional.recomputed_forward`` and does not."""
  e = w_gate.shape[0]
  f = w_down.shape[1]
  from .functional import _native, in_recomputed_forward, inference_only
  ok = (_kernels_ok(x, w_gate, w_down) and x.shape[-1] % 64 == 0 and f % 64 == 0 and x.is_cuda)
  if ok:
    if (capacity is None and e <= 256 and inference_only() and not in_recomputed_forward()
        and all(w.is_contiguous() and w.data_ptr() % 16 == 0 for w in (w_gate, w_up, w_down) if w is not None)):
      align = few_rows_align(*idx.shape, e)
      if align is not None:
        if (nat := _native()) is not None and not _debug.bounds_enabled():
          y = nat.grouped_mlp_few_rows(x, weights, idx, w_gate, w_up, w_down, fused_gate_up, align)
          if y is not None:
            return y
        return grouped_mlp_few_rows(x.contiguous(), weights.float().contiguous(), idx, w_gate, w_up, w_down,
                                    fused_gate_up, align)
    plan = build_dispatch_plan(idx, e, capacity, rows_per_group)
    wu = w_gate if fused_gate_up else w_up
    return _GroupedMLPFn.apply(x.contiguous(), weights.float().contiguous(), w_gate, wu, w_down, plan, fused_gate_up)
  dropped = None
  if capacity is not None:
    dropped = build_dispatch_plan(idx, e, capacity, rows_per_group).dest < 0
  return grouped_mlp_reference(x, weights, idx, w_gate, w_up, w_down, fused_gate_up, dropped)
