"""The native operators (csrc/torch_ops.cpp) give what the Python definitions give, call by call, and leave to those
whatever they are not meant for."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.ops import _lib, moe
from torchprime_b200.ops import functional as ops

BF = torch.bfloat16


def _r(*shape, grad=False, seed=0, dtype=BF):
  g = torch.Generator("cuda").manual_seed(seed + sum(shape))
  return torch.randn(*shape, device="cuda", generator=g).to(dtype).requires_grad_(grad)


def _adjacent(*shapes, grads):
  flat = _r(sum(a * b for a, b in shapes)) / 16
  out, at = [], 0
  for (a, b), g in zip(shapes, grads):
    out.append(flat[at:at + a * b].view(a, b).detach().requires_grad_(g))
    at += a * b
  return out


def _tables(s, half):
  a = torch.arange(s, device="cuda", dtype=torch.float32)[:, None] / torch.arange(1, half + 1, device="cuda")
  return a.cos(), a.sin()


def _linear(n, grads, residual, shape=(2, 19, 64)):
  def call():
    x = _r(*shape, grad=grads[0])
    ws = _adjacent(*[(64, 64), (32, 64), (8, 64)][:n], grads=grads[1:1 + n])
    rows = sum(w.shape[0] for w in ws)
    res = _r(*shape[:-1], rows, grad=grads[-1], seed=3) if residual else None
    return ops.linear(x, ws if n > 1 else ws[0], residual=res), [x, *ws, res]
  return call


def _swiglu(grads):
  def call():
    x, ws = _r(3, 40, 64, grad=grads[0]), _adjacent((72, 64), (72, 64), grads=grads[1:])
    return ops.linear_swiglu(x, *ws), [x, *ws]
  return call


def _norm(fn, dims, grads=(True, True)):
  def call():
    x, w = _r(*dims, grad=grads[0]), _r(dims[-1], grad=grads[1])
    return fn(x, w, 1e-5), [x, w]
  return call


def _rope(pos, interleaved, col0, stride):
  def call():
    x = _r(2, 30, 4 * 192, grad=True)
    p = torch.randint(0, 40, (60,), device="cuda", dtype=torch.int32) if pos else None
    if p is not None:
      p = (torch.arange(60, device="cuda") * 7 % 40).to(torch.int32)
    cos, sin = _tables(40, 32)
    return ops.rope_slices(x * 1, cos, sin, 4, 64, 30, col0, stride, pos=p, interleaved=interleaved), [x]
  return call


def _qkv(s, seg, pos, window, causal=True):
  def call():
    x = _r(2, s, 6 * 128, grad=True)
    ids = (torch.arange(s, device="cuda") // 77).expand(2, s) if seg else None
    p = (torch.arange(2 * s, device="cuda") % s).to(torch.int32) if pos else None
    return ops.attention_qkv(x, 4, 1, 128, causal=causal, window=window, q_segment_ids=ids, q_positions=p), [x]
  return call


def _attn(dqk, sq, sk, seg=False, softcap=None, sliced=False):
  def call():
    q, k, v = _r(2, sq, 4, dqk, grad=True), _r(2, sk, 2, dqk, grad=True), _r(2, sk, 2, 128, grad=True)
    inputs = [q, k, v]
    if sliced:
      kv = _r(2, sk, 2, dqk + 128, grad=True)
      k, v, inputs = kv[..., :dqk].contiguous(), kv[..., dqk:].contiguous(), [q, kv]
    ids = (torch.arange(sq, device="cuda") // 100).expand(2, sq).contiguous() if seg else None
    return ops.attention(q, k, v, causal=True, scale=0.07, q_segment_ids=ids, softcap=softcap), inputs
  return call


def _latent():
  x = _r(2, 21, 96 + 64, grad=True)
  lat, rot = ops.latent_split(x, 96)
  return (lat, rot), [x]


def _latent_rope(pos, interleaved):
  def call():
    x = _r(2, 30, 96 + 64, grad=True)
    cos, sin = _tables(40, 32)
    p = (torch.arange(60, device="cuda") * 7 % 40).to(torch.int32) if pos else None
    return ops.latent_split_rope(x * 1, 96, cos, sin, 30, pos=p, interleaved=interleaved), [x]
  return call


def _pack():
  kv, rot = _r(2, 21, 3 * (64 + 128), grad=True), _r(2, 21, 64, grad=True)
  return ops.mla_pack(kv, rot, 3, 64, 128), [kv, rot]


CALLS = {
  "linear": _linear(1, (True, True, False), False),
  "linear input only": _linear(1, (True, False, False), False),
  "linear weight only": _linear(1, (False, True, False), False),
  "linear residual": _linear(1, (True, True, True), True),
  "linear frozen residual": _linear(1, (False, True, False), True),
  "linear residual only": _linear(1, (False, False, True), True),
  "linear of three": _linear(3, (True, True, True, True, False), False),
  "linear of three, one frozen": _linear(3, (True, True, False, True, True), True),
  "linear of two": _linear(2, (False, False, True, False), False),
  "linear 2-D": _linear(1, (True, True, True), True, shape=(200, 64)),
  "linear without grads": _linear(2, (False, False, False, False), True),
  "swiglu": _swiglu((True, True, True)),
  "swiglu weights": _swiglu((False, True, True)),
  "swiglu input": _swiglu((True, False, False)),
  "norm": _norm(ops.rms_norm, (2, 30, 264)),
  "norm input": _norm(ops.rms_norm, (30, 64), (True, False)),
  "norm weight": _norm(ops.rms_norm, (1, 500, 2048), (False, True)),
  "norm pass": _norm(ops.rms_norm_residual, (2, 30, 264)),
  "norm pass wide": _norm(ops.rms_norm_residual, (300, 8192)),
  "rope": _rope(False, False, 0, 64),
  "rope slices": _rope(True, True, 128, 192),
  "qkv": _qkv(130, False, False, None),
  "qkv segments": _qkv(300, True, False, None),
  "qkv positions, window": _qkv(200, True, True, 50),
  "qkv full": _qkv(65, False, False, None, causal=False),
  "attention": _attn(128, 100, 100),
  "attention wide": _attn(192, 200, 200, sliced=True),
  "attention fewer queries": _attn(128, 60, 200),
  "attention segments": _attn(192, 300, 300, seg=True),
  "attention cap": _attn(128, 140, 140, softcap=20.0),
  "latent": _latent,
  "latent, rotated": _latent_rope(False, True),
  "latent, rotated halves": _latent_rope(True, False),
  "pack": _pack,
}


def _run(call, backward=True):
  y, inputs = call()
  ys = list(y) if isinstance(y, tuple) else [y]
  inputs = [t for t in inputs if t is not None and t.requires_grad]
  grads = []
  if backward and inputs and any(t.requires_grad for t in ys):
    grads = torch.autograd.grad([t for t in ys if t.requires_grad], inputs,
                                [_r(*t.shape, seed=11 + i) for i, t in enumerate(ys) if t.requires_grad], allow_unused=True)
  return [t.detach() for t in ys], list(grads)


@pytest.fixture
def in_python(monkeypatch):
  _lib.lib()
  return lambda: monkeypatch.setattr(_lib, "_native", None)


@pytest.mark.parametrize("name", CALLS)
def test_same_as_the_python_definition(cuda_lib, in_python, monkeypatch, name):
  _lib.lib()
  before = _lib._native.launch_count()
  got = _run(CALLS[name])
  with torch.no_grad():
    bare = _run(CALLS[name], backward=False)[0]
  assert _lib._native.launch_count() > before or name == "latent"
  in_python()
  want = _run(CALLS[name])
  assert len(got[1]) == len(want[1])
  for a, b, c in zip(got[0], want[0], bare):
    assert torch.equal(a, b) and torch.equal(a, c) and a.stride() == b.stride()
  for a, b in zip(got[1], want[1]):
    assert (a is None) == (b is None)
    # (the norm's weight gradient is a sum by atomics, which does not repeat itself to the last bit)
    if a is not None:
      assert a.dtype == b.dtype and torch.allclose(a, b, rtol=1e-2, atol=0) if "norm" in name else torch.equal(a, b)


def test_saved_tensor_hooks_and_checkpoints_see_the_native_nodes(cuda_lib):
  _lib.lib()
  x, w = _r(40, 64, grad=True), (_r(64, 64) / 8).requires_grad_(True)
  packed = []
  with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
    y = ops.linear(ops.rms_norm(x, w[0].detach(), 1e-5), w)
  assert len(packed) >= 4
  want = torch.autograd.grad(ops.linear(ops.rms_norm(x, w[0].detach(), 1e-5), w), (x, w), torch.ones_like(y))
  for a, b in zip(torch.autograd.grad(y, (x, w), torch.ones_like(y)), want):
    assert torch.equal(a, b)
  z = torch.utils.checkpoint.checkpoint(lambda t: ops.linear_swiglu(t, w[:32], w[32:]), x, use_reentrant=False)
  plain = ops.linear_swiglu(x, w[:32], w[32:])
  for a, b in zip(torch.autograd.grad(z.sum(), (x, w)), torch.autograd.grad(plain.sum(), (x, w))):
    assert torch.equal(a, b)


def test_a_saved_input_that_was_changed_is_noticed(cuda_lib):
  _lib.lib()
  x, w = _r(40, 64), (_r(64, 64) / 8).requires_grad_(True)
  y = ops.linear(x, w)
  x.add_(1)
  with pytest.raises(RuntimeError, match="modified by an inplace operation"):
    y.sum().backward()


def test_main_grad(cuda_lib):
  """Weights that collect their gradients keep the Python definition; so do the gradients of weights that are told to
  after the forward pass."""
  _lib.lib()
  x = _r(40, 64, grad=True)
  ws, nw = _adjacent((64, 64), (32, 64), grads=(True, True)), _r(64, grad=True)
  want = torch.autograd.grad(ops.linear(ops.rms_norm(x, nw, 1e-5), ws).sum(), [nw, *ws])
  sink = torch.zeros(96, 64, device="cuda", dtype=torch.float32)
  for when in ("before", "after"):
    sink.zero_()
    params = [torch.nn.Parameter(t.detach()) for t in (nw, *ws)]
    def attach():
      params[0].main_grad = torch.zeros(64, device="cuda")
      params[1].main_grad, params[2].main_grad = sink[:64], sink[64:]
    if when == "before":
      attach()
    loss = ops.linear(ops.rms_norm(x, params[0], 1e-5), params[1:]).sum()
    if when == "after":
      attach()
    loss.backward()
    assert all(p.grad is None for p in params)
    for p, b in zip(params, want):
      assert torch.allclose(p.main_grad, b.float(), rtol=2e-2, atol=1e-2)


def test_what_is_not_meant_for_them(cuda_lib):
  _lib.lib()
  nat = _lib._native
  x, w = _r(40, 64), _r(64, 64)
  assert nat.linear(x, w, None) is not None
  for bad in (x.float(), x.cpu(), x[:, :32], x[:0], x[..., :60].contiguous(), 3.0, None):
    assert nat.linear(bad, w, None) is None
  assert nat.linear(x, w.t(), None) is None and nat.linear(x, w[:60], None) is None
  assert nat.linear(x, [w[:32], w[40:]], None) is None and nat.linear(x, [], None) is None
  assert nat.linear(x, w, x.float()) is None and nat.linear(x, w, x[:20]) is None
  assert nat.rms_norm(x, w[:, 0], 1e-5) is None and nat.rms_norm(x, w[0, :32], 1e-5) is None
  with torch.autograd.forward_ad.dual_level():
    assert nat.linear(x, w, None) is None
  torch.func.vmap(lambda t: (_assert_none(nat.linear(t, w, None)), t)[1])(x[None])
  torch.func.grad(lambda t: (_assert_none(nat.rms_norm(t, w[0], 1e-5)), t.float().sum())[1])(x)
  from torch.utils._python_dispatch import TorchDispatchMode
  class Watch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
      return func(*args, **(kwargs or {}))
  with Watch():
    assert nat.linear(x, w, None) is None
  with ops.backend("torch"):
    assert ops._native() is None


def _assert_none(v):
  assert v is None


def test_refused_arguments_raise_the_same_error(cuda_lib):
  _lib.lib()
  x = torch.empty(40 * 64 + 1, device="cuda", dtype=BF)[1:].view(40, 64)      # not 16-byte aligned
  w = (_r(64, 64) / 8).requires_grad_(True)
  with pytest.raises(_lib.KernelError):
    ops.linear(x, w)
  y = ops.linear(x.clone(), w)
  dy = torch.empty(40 * 64 + 1, device="cuda", dtype=BF)[1:].view(40, 64)
  with pytest.raises(_lib.KernelError):                                       # from the engine's thread
    y.backward(dy)


@pytest.mark.parametrize("tokens,fused", [(1, False), (7, False), (30, True)])
def test_experts_without_gradients(cuda_lib, in_python, tokens, fused):
  _lib.lib()
  e, d, f, k = 16, 128, 64, 4
  x, wd = _r(tokens, d), _r(e, f, d) / 8
  wg, wu = _r(e, d, 2 * f if fused else f) / 11, None if fused else _r(e, d, f, seed=5) / 11
  logits = _r(tokens, e, dtype=torch.float32)
  def call():
    with torch.no_grad():
      w, idx, scores = moe.router_topk(logits, k, mode="sigmoid", bias=torch.ones(e, device="cuda"), scale=2.0)
      return [w, idx, scores, moe.grouped_mlp(x, w, idx, wg, wu, wd, fused_gate_up=fused),
              ops.linear_f32(x, wd[0]) if f % 8 == 0 and d == wd.shape[2] else x]
  got = call()
  in_python()
  for a, b in zip(got, call()):
    assert torch.equal(a, b)


@pytest.mark.parametrize("window,scale,softcap", [(70.0, None, None), (np.int64(70), np.float32(0.25), None),
                                                  (None, torch.tensor(0.25), 30), (70, 1, 30.0)])
def test_options_given_as_other_numbers(cuda_lib, window, scale, softcap):
  """What int() and float() take is taken, as by the Python definitions."""
  _lib.lib()
  plain = dict(window=None if window is None else int(window), scale=None if scale is None else float(scale))
  cap = None if softcap is None else float(softcap)
  q, k, v = _r(1, 100, 4, 128), _r(1, 100, 2, 128, seed=1), _r(1, 100, 2, 128, seed=2)
  assert torch.equal(ops.attention(q, k, v, window=window, scale=scale, softcap=softcap),
                     ops.attention(q, k, v, softcap=cap, **plain))
  x = _r(1, 100, 8 * 128)
  assert torch.equal(ops.attention_qkv(x, 4, 2, 128, window=window, scale=scale), ops.attention_qkv(x, 4, 2, 128, **plain))


def _steps(seed, n=6):
  """A few operators, forward and backward, in the current stream; what they give in the end."""
  x = _r(2, 130, 256, grad=True, seed=seed)
  ws = _adjacent((192, 256), (192, 256), grads=(True, True))
  wd, wn, wq = _r(256, 192, grad=True, seed=1), _r(256, grad=True, seed=2), _r(6 * 128, 256, grad=True, seed=3)
  cos, sin = _tables(130, 64)
  leaves = [x, *ws, wd, wn, wq]
  for t in leaves:
    t.grad = None
  for _ in range(n):
    h, res = ops.rms_norm_residual(x, wn, 1e-5)
    qkv = ops.rope_inplace(ops.linear(h, wq / 16), cos, sin, 5, 128, 130)
    a = ops.attention_qkv(qkv, 4, 1, 128)
    y = ops.swiglu_mlp(h, *ws, wd, res) + a.view(2, 130, 512)[..., :256]
    y.backward(torch.linspace(-1, 1, y.numel(), device="cuda").view(y.shape).to(BF))
  return [y.detach()] + [t.grad for t in leaves if t is not wn]      # (the norm's weight gradient is summed by atomics)


def test_streams_and_threads(cuda_lib):
  """Several threads, each in a stream of its own, give what one gives alone in the default stream."""
  import threading
  want = [_steps(s) for s in range(3)]
  torch.cuda.synchronize()
  got, errors = {}, []
  def work(s):
    try:
      stream = torch.cuda.Stream()
      with torch.cuda.stream(stream):
        for _ in range(3):
          got[s] = _steps(s)
      stream.synchronize()
    except BaseException as e:      # noqa: BLE001
      errors.append(e)
  threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
  for t in threads:
    t.start()
  for t in threads:
    t.join()
  assert not errors, errors
  for s in range(3):
    for a, b in zip(got[s], want[s]):
      assert torch.equal(a, b)


@pytest.mark.parametrize("b,s", [(3, 1), (2, 2)])
@pytest.mark.parametrize("native", [True, False])
def test_one_token_per_row(cuda_lib, in_python, b, s, native):
  """A fused projection of one token per row: every batch finds its own heads."""
  _lib.lib()
  if not native:
    in_python()
  x = _r(b, s, 6 * 128, grad=True)
  y = ops.attention_qkv(x, 4, 1, 128, causal=False)
  y.sum().backward()
  for i in range(b):
    one = x.detach()[i:i + 1].clone().requires_grad_(True)
    z = ops.attention_qkv(one, 4, 1, 128, causal=False)
    z.sum().backward()
    assert torch.equal(y[i:i + 1], z) and torch.equal(x.grad[i:i + 1], one.grad)
