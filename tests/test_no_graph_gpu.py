"""Operators with nothing recorded."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import functional as ops


def test_operators_without_a_graph_equal_those_with_one(cuda_lib):
  """Nothing recorded: the operators skip their autograd functions; results, in-place writes and version
  counters are the same."""
  torch.manual_seed(0)
  x = torch.randn(2, 40, 256, device="cuda", dtype=torch.bfloat16)
  w = torch.randn(256, 256, device="cuda", dtype=torch.bfloat16) / 16
  g = torch.randn(512, 256, device="cuda", dtype=torch.bfloat16) / 16
  n = torch.randn(256, device="cuda", dtype=torch.bfloat16)
  ids = torch.randint(0, 256, (2, 40), device="cuda")
  cos, sin = torch.randn(40, 64, device="cuda"), torch.randn(40, 64, device="cuda")
  def every():
    qkv = torch.randn(2, 40, 6 * 128, device="cuda", dtype=torch.bfloat16, generator=torch.Generator("cuda").manual_seed(1))
    r = ops.rope_inplace(qkv * 1, cos, sin, 5, 128, 40)
    return [ops.linear(x, w), ops.linear(x, w, residual=x), ops.linear_swiglu(x, g[:256], g[256:]), ops.rms_norm(x, n, 1e-5),
            *ops.rms_norm_residual(x, n, 1e-5), r, ops.embedding(ids, w),
            ops.attention_qkv(r, 4, 1, 128)]
  with_graph = every()
  with torch.no_grad():
    without = every()
  for a, b in zip(with_graph, without):
    assert torch.equal(a, b) and not b.requires_grad
  t = torch.randn(1, 40, 256, device="cuda", dtype=torch.bfloat16)
  v = t._version
  with torch.no_grad():
    assert ops.rope_inplace(t, cos, sin, 2, 128, 40) is t and t._version == v + 1
  with torch.inference_mode():
    ops.rope_inplace(torch.randn(1, 40, 256, device="cuda", dtype=torch.bfloat16), cos, sin, 2, 128, 40)


def test_fused_projection_with_a_row_pitch(cuda_lib):
  """A projection that is a slice of wider rows gives the same result with and without a graph."""
  from torchprime_b200.ops import attention_sm100 as A
  qkv = torch.randn(2, 70, 6 * 128 + 64, device="cuda", dtype=torch.bfloat16)[..., :6 * 128]
  with_graph = A.attention_qkv(qkv, 4, 1, 128)
  with torch.no_grad():
    assert torch.equal(A.attention_qkv(qkv, 4, 1, 128), with_graph)
    assert torch.equal(A.attention_qkv(qkv.contiguous(), 4, 1, 128), with_graph)


@pytest.mark.parametrize("op", ["linear", "swiglu", "norm", "embedding", "attention", "segments", "router"])
def test_traces_follow_their_input(cuda_lib, op):
  """An operator traced with nothing recorded computes from the input of each call."""
  from torchprime_b200.ops import moe
  torch.manual_seed(0)
  w = torch.randn(128, 64, device="cuda", dtype=torch.bfloat16) / 8
  ids = torch.arange(300, device="cuda")[None] // 70
  fn, shape = {
    "linear": (lambda x: ops.linear(x, w), (30, 64)),
    "swiglu": (lambda x: ops.linear_swiglu(x, w[:64], w[64:]), (30, 64)),
    "norm": (lambda x: ops.rms_norm(x, w[0], 1e-5), (30, 64)),
    "embedding": (lambda x: ops.embedding((x[:, 0].float().abs() * 10).long().clamp(0, 127), w), (30, 64)),
    "attention": (lambda x: ops.attention_qkv(x, 4, 1, 128), (1, 40, 6 * 128)),
    "segments": (lambda x: ops.attention_qkv(x, 4, 1, 128, q_segment_ids=ids), (1, 300, 6 * 128)),
    "router": (lambda x: moe.router_topk(x.float(), 6)[0], (30, 64)),
  }[op]
  first, second = (torch.randn(*shape, device="cuda", dtype=torch.bfloat16) for _ in range(2))
  with torch.no_grad():
    traced = torch.jit.trace(fn, (first,), check_trace=False)
    assert torch.equal(traced(second), fn(second)) and torch.equal(traced(first), fn(first))
