"""One cached decode step of latent attention (csrc/mla_decode.cu): rotary embedding, latent norm and
cache update, query folding through the key up-projection, attention over the compressed cache and the
value up-projection, in four launches.
"""

from __future__ import annotations

from ctypes import c_float, c_int, c_longlong, c_void_p

import torch

from . import _lib
from ._lib import check, lib, ptr, stream_ptr

P, I, LL, F = c_void_p, c_int, c_longlong, c_float
_lib.register_signature("tpb_mla_decode_ranges", [I, I, I])
_lib.register_signature("tpb_mla_decode", [P, P, P, P, P, P, P, LL, LL, P, P, P, P, P, I, I, I, I, I, I, I, F, F, I, I,
                                           P])


def _rows(t, width) -> bool:
  return t.is_contiguous() and t.shape[-1] == width and t.data_ptr() % 16 == 0


def supported(q, ckv, norm_w, kv_cache, pe_cache, w, heads, dn, dr, dv, c) -> bool:
  """One token per sequence, bf16 throughout, rotary width 64, a latent of at most 512 values, value width up to 4096
  and as many sequences as a grid dimension holds."""
  from .functional import _native, inference_only, use_kernels
  if (nat := _native()) is not None and nat.absorb_supported(q, ckv, norm_w, kv_cache, pe_cache, w, heads, dn, dr, dv, c):
    return True
  ts = (q, ckv, norm_w, kv_cache, pe_cache, w)
  if not all(t.is_cuda and t.dtype == torch.bfloat16 for t in ts) or not use_kernels(*ts):
    return False
  return (q.shape[1] == 1 and q.shape[0] <= 65535 and dv <= 4096 and dr == 64 and c % 64 == 0 and 64 <= c <= 512 and dn % 8 == 0 and 8 <= dn <= 512
          and _rows(q, heads * (dn + dr)) and _rows(ckv, c + dr) and _rows(norm_w, c) and _rows(w, c)
          and w.numel() == heads * (dn + dv) * c and _rows(kv_cache, c) and _rows(pe_cache, dr)
          and inference_only())


def absorb_step(q, ckv, norm_w, eps, cos, sin, pos, kv_cache, pe_cache, w, heads, dn, dv, scale, interleaved):
  """q [B, 1, heads * (dn + 64)] (its rotary part is rotated in place), ckv [B, 1, C + 64]; the token's
  normalised latent and rotated key go to position ``pos`` of the caches [>=B, S, C] / [>=B, S, 64] and it
  attends to positions 0 .. pos.  ``w``: the key / value up-projection [heads * (dn + dv), C].
  Returns [B, 1, heads * dv]."""
  from .functional import _native
  if (nat := _native()) is not None:
    o = nat.absorb_step(q, ckv, norm_w, eps, cos, sin, pos, kv_cache, pe_cache, w, heads, dn, dv, scale, interleaved)
    if o is not None:
      return o
  b, c = q.shape[0], kv_cache.shape[-1]
  assert cos.dtype == sin.dtype == torch.float32 and cos.is_contiguous() and sin.is_contiguous()
  assert cos.shape[0] > pos and cos.shape[1] == 32 and kv_cache.shape[1] > pos and kv_cache.shape[0] >= b
  out = torch.empty(b, 1, heads * dv, dtype=q.dtype, device=q.device)
  ranges = lib().tpb_mla_decode_ranges(b, heads, pos + 1)
  scratch = torch.empty(b * heads * (c + ranges * (c + 2)), dtype=torch.float32, device=q.device)
  base = scratch.data_ptr()
  part_o = base + 4 * b * heads * c
  part_ml = part_o + 4 * b * heads * ranges * c
  rc = lib().tpb_mla_decode(ptr(q), ptr(ckv), ptr(norm_w), ptr(cos), ptr(sin), ptr(kv_cache), ptr(pe_cache),
                            kv_cache.stride(0), pe_cache.stride(0), ptr(w), ptr(out), base, part_o, part_ml, b, heads, dn,
                            dv, c, pe_cache.shape[-1], pos, float(scale), float(eps), int(interleaved), ranges,
                            stream_ptr())
  check(rc, f"mla_decode B={b} H={heads} pos={pos}")
  return out
