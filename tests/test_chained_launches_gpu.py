"""Chained launches (csrc/common.cuh, chain_launch / chain_wait)."""

import time

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import _lib, kernels as k
from torchprime_b200.parallel import fsdp_comm      # noqa: F401  (declares the gather's entry points)


@pytest.mark.parametrize("m,n,kk", [(8192, 16384, 16384), (2048, 1152, 131072)])      # CTA pairs, single CTAs
def test_no_kernel_moves_in_behind_a_gemm_that_may_wait_for_a_gather(cuda_lib, m, n, kk):
  """While a GEMM that waits in-kernel for gathered weights runs, a kernel on another stream (the one that publishes a
  shard, in a real gather) can start, although a chained kernel is queued behind the GEMM.  Nothing here waits for that
  kernel: every shard is published beforehand, and what is looked at is when it ran."""
  L = _lib.lib()
  a = torch.randn(m, kk, device="cuda").to(torch.bfloat16)
  w = (torch.randn(n, kk, device="cuda") / 128).to(torch.bfloat16)
  out = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
  chunk = 1 << 20
  flags = torch.full(((n * kk + chunk - 1) // chunk,), 1, device="cuda", dtype=torch.int32)
  cos, sin = torch.ones(2048, 64, device="cuda"), torch.zeros(2048, 64, device="cuda")
  shard, side = torch.zeros(1, device="cuda", dtype=torch.int32), torch.cuda.Stream()
  for _ in range(2):      # (the first round loads the kernels)
    torch.cuda.synchronize()
    first, last, ran = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    first.record()
    _lib.check(L.tpb_gemm_ag_wait_bf16(a.data_ptr(), out.data_ptr(), m, n, kk, kk, n, k.EPI_BF16, None, 0, None, 0,
                                       w.data_ptr(), 0, 1, n * kk, chunk, flags.data_ptr(), 1, _lib.stream_ptr()), "gemm")
    k.rope_(out, 0, n // 128, 128, cos, sin, 2048)      # a chained kernel with CTAs for every SM; rotates by nothing
    time.sleep(1e-4)      # (time for that kernel's CTAs to move in, were they let in)
    with torch.cuda.stream(side):
      _lib.check(L.tpb_flag_set(shard.data_ptr(), 7, _lib.stream_ptr()), "flag_set")
      ran.record()
    last.record()
    torch.cuda.synchronize()
  assert int(shard) == 7
  whole, left = first.elapsed_time(last), ran.elapsed_time(last)
  assert whole > 0.4 and left > 0.4 * whole, f"the other stream's kernel ended {left:.2f} ms before the {whole:.2f} ms were over"
  want = a[:64].double() @ w.double().t()
  assert bool(((out[:64].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-6 * kk).all())
