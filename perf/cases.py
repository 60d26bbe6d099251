"""The work this framework is used for, as timed cases: decoder blocks and heads of the model
families in ``torchprime_b200/configs/model`` in training, evaluation and cached inference.

Every case goes through a module or operator that a program can call.  Weights that the FSDP
engine keeps back to back in a unit's flat buffer (q/k/v, gate/up) lie back to back here too.
``exact`` restates the same mathematics in 64-bit plain PyTorch.
"""

import math

import torch
import torch.nn.functional as F

from torchprime_b200.config import compose
from torchprime_b200.experimental.deepseek_inference.engine import DeepseekInferenceEngine
from torchprime_b200.models.deepseek_v3 import DeepseekV3Attention, DeepseekV3ForCausalLM, DeepseekV3MoE
from torchprime_b200.models.llama import CausalLMHead, LlamaDecoderLayer, LlamaRMSNorm
from torchprime_b200.models.model_utils import set_default_dtype
from torchprime_b200.ops import functional as ops
from torchprime_b200.ops import moe as moe_ops

BF16 = torch.bfloat16
ENGINE_LAYERS = 3          # dense layers of the cached-inference model (see listed())


# ------------------------------------------------------------------------------- the cases
def listed():
  return [
    # Evaluating or scoring one short sequence: a decoder layer of Llama-3-8B, weight-bound.
    {"name": "layer_eval_short", "kind": "layer_eval", "batch": 1, "seq": 77},
    # The ordinary training block: the same layer forward and backward at 4096 tokens.
    {"name": "layer_train", "kind": "layer_train", "batch": 1, "seq": 4096},
    # Long-context pre-training: causal attention of the benchmark's sequence length.
    {"name": "attn_train_long", "kind": "attn_train", "batch": 1, "seq": 8192, "heads": 32, "kv_heads": 8,
     "segments": 0},
    # Supervised fine-tuning: packed conversations of ragged lengths, masked by segment ids.
    {"name": "attn_train_packed", "kind": "attn_train", "batch": 2, "seq": 1999, "heads": 32, "kv_heads": 8,
     "segments": 7},
    # Final norm, 128k-vocabulary head and loss of a ragged batch, forward and backward.
    {"name": "head_train", "kind": "head_train", "tokens": 3001},
    # Mixtral-8x7B's routed experts in training (few experts, wide FFN).
    {"name": "moe_train_wide", "kind": "moe_train_wide", "tokens": 4096},
    # DeepSeek-V2-Lite's MoE block in training (64 narrow experts, router and shared experts).
    {"name": "moe_train_fine", "kind": "moe_train_fine", "batch": 1, "seq": 1500},
    # The same block inside a decode step of four sequences.
    {"name": "moe_decode", "kind": "moe_decode", "batch": 4, "seq": 1},
    # DeepSeek-V2-Lite's latent attention in training.
    {"name": "mla_train", "kind": "mla_train", "batch": 1, "seq": 2048},
    # One cached decode step of four sequences; the model is three dense layers and the head, so
    # that its logits do not hang on a near-tie of a router (the routed block has its own case).
    {"name": "decode_step", "kind": "decode", "batch": 4, "start": 1500},
    # Prefill of a prompt through the same engine with the uncompressed cache.
    {"name": "prefill", "kind": "prefill", "batch": 1, "seq": 900},
    # A norm with its residual connection, forward and backward, at the benchmark's size.
    {"name": "norm_train", "kind": "norm_train", "tokens": 8192, "dim": 4096},
  ]


def _log_int(rng, lo, hi):
  return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
  kind = rng.choice(["layer_eval", "layer_train", "attn_train", "head_train", "moe_train_wide", "moe_train_fine",
                     "moe_decode", "mla_train", "decode", "prefill", "norm_train"])
  if kind == "layer_eval":
    return {"kind": kind, "batch": rng.randint(1, 4), "seq": _log_int(rng, 1, 700)}
  if kind == "layer_train":
    b = rng.randint(1, 2)
    return {"kind": kind, "batch": b, "seq": _log_int(rng, 33, 4096 // b)}
  if kind == "attn_train":
    b = rng.randint(1, 4)
    h, hkv = rng.choice([(32, 8), (40, 8), (64, 8), (16, 16)])
    s = _log_int(rng, 40, min(8192, 12000 // b))
    return {"kind": kind, "batch": b, "seq": s, "heads": h, "kv_heads": hkv, "segments": rng.choice([0, 0, 3, 9])}
  if kind in ("head_train", "moe_train_wide"):
    return {"kind": kind, "tokens": _log_int(rng, 60, 3000 if kind == "head_train" else 4000)}
  if kind in ("moe_train_fine", "mla_train"):
    b = rng.randint(1, 3)
    return {"kind": kind, "batch": b, "seq": _log_int(rng, 50, 4000 // b)}
  if kind == "moe_decode":
    return {"kind": kind, "batch": rng.randint(1, 16), "seq": 1}
  if kind == "decode":
    return {"kind": kind, "batch": rng.randint(1, 8), "start": _log_int(rng, 20, 3500)}
  if kind == "prefill":
    return {"kind": kind, "batch": rng.randint(1, 2), "seq": _log_int(rng, 128, 1500)}
  return {"kind": kind, "tokens": _log_int(rng, 60, 12000), "dim": rng.choice([2048, 4096, 5120])}


# ------------------------------------------------------------------------------- inputs
def _config(name, **changes):
  cfg = compose("default", [f"model={name}"]).model
  for k, v in changes.items():
    cfg[k] = v
  return cfg


def _gen(seed):
  return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=BF16):
  return torch.empty(*shape, device="cuda", dtype=dtype).normal_(0.0, std, generator=g)


def _lay_out(*weights):
  """Put the weights back to back in one buffer, as the FSDP engine's flat units do."""
  flat = torch.cat([w.detach().reshape(-1) for w in weights])
  at = 0
  for w in weights:
    w.data = flat[at:at + w.numel()].view(w.shape)
    at += w.numel()


def _init(module, g):
  """Norm weights near one, matrices N(0, 0.02), in parameter order."""
  for p in module.parameters():
    if p.dim() == 1:
      p.data.normal_(1.0, 0.05, generator=g)
    else:
      p.data.normal_(0.0, 0.02, generator=g)
  for m in module.modules():
    if hasattr(m, "gate_proj"):
      _lay_out(m.gate_proj.weight, m.up_proj.weight)
    if hasattr(m, "k_proj"):
      _lay_out(m.q_proj.weight, m.k_proj.weight, m.v_proj.weight)
  return module


def _build(cls, *args):
  with set_default_dtype(BF16), torch.device("cuda"):
    return cls(*args).to("cuda")


def _tables(positions, inv_freq):
  ang = torch.arange(positions, dtype=torch.float64)[:, None] * inv_freq[None, :]
  return ang.cos().float().cuda(), ang.sin().float().cuda()


def _plain_inv_freq(dim, theta):
  return theta ** (-torch.arange(0, dim, 2, dtype=torch.float64) / dim)


def _yarn_inv_freq(cfg):
  """YaRN frequencies of the rotary part of a latent-attention model (published definition)."""
  rs, dim, base = cfg.rope_scaling, cfg.qk_rope_head_dim, float(cfg.rope_theta)
  orig = rs["original_max_position_embeddings"]
  factor = cfg.max_position_embeddings / orig
  edge = lambda rot: dim * math.log(orig / (rot * 2 * math.pi)) / (2 * math.log(base))  # noqa: E731
  low, high = max(math.floor(edge(rs["beta_fast"])), 0), min(math.ceil(edge(rs["beta_slow"])), dim - 1)
  ramp = ((torch.arange(dim // 2, dtype=torch.float64) - low) / max(high - low, 1e-3)).clamp(0, 1)
  plain = _plain_inv_freq(dim, base)
  return plain / factor * ramp + plain * (1 - ramp)


def _segments(case, g):
  """Ragged lengths of packed conversations: ids that do not decrease along the sequence."""
  if not case["segments"]:
    return None
  cuts = torch.randint(0, case["seq"], (case["batch"], case["segments"] - 1), device="cuda", generator=g)
  at = torch.arange(case["seq"], device="cuda")
  return (at[None, :, None] >= cuts[:, None, :]).sum(-1).to(torch.int32)


def _decided(x, gate, k):
  """Tokens whose k-th and (k+1)-th expert are a tie to within rounding take another token's place, so
  that every correct router makes the same choices."""
  flat = x.view(-1, x.shape[-1])
  top = (flat.double() @ gate.detach().double().t()).topk(k + 1, dim=-1)[0]
  gap = top[:, k - 1] - top[:, k]
  return torch.where((gap < 1e-4)[:, None], flat[gap.argmax()], flat).view_as(x)


def _llama_like(case, g):
  cfg = _config("llama-3-8b")
  layer = _init(_build(LlamaDecoderLayer, cfg, 0), g)
  cos, sin = _tables(case["seq"], _plain_inv_freq(128, float(cfg.rope_theta)))
  x = _randn(g, case["batch"], case["seq"], cfg.hidden_size)
  return {"cfg": cfg, "layer": layer, "cos": cos, "sin": sin, "x": x}


def prepare(case, seed):
  kind, g = case["kind"], _gen(seed)
  st = {"kind": kind}
  if kind in ("layer_eval", "layer_train"):
    st.update(_llama_like(case, g))
  elif kind == "attn_train":
    h, hkv = case["heads"], case["kv_heads"]
    st.update(h=h, hkv=hkv, x=_randn(g, case["batch"], case["seq"], (h + 2 * hkv) * 128), seg=_segments(case, g))
    st["dy"] = _randn(g, case["batch"], case["seq"], h, 128)
  elif kind == "head_train":
    cfg = _config("llama-3-8b")
    norm = _build(LlamaRMSNorm, cfg.hidden_size, cfg.rms_norm_eps)
    head = _build(lambda: torch.nn.Linear(cfg.hidden_size, cfg.vocab_size, bias=False))
    st["layer"] = _init(_build(CausalLMHead, norm, head, cfg.vocab_size), g)
    st["x"] = _randn(g, 1, case["tokens"], cfg.hidden_size)
    tg = torch.randint(0, cfg.vocab_size, (1, case["tokens"]), device="cuda", generator=g)
    skip = torch.rand(1, case["tokens"], device="cuda", generator=g) < 0.1
    skip[0, 0] = False
    st["targets"] = tg.masked_fill(skip, -100)
  elif kind == "moe_train_wide":
    cfg = _config("mixtral-8x7b")
    e, d, f, t = cfg.num_local_experts, cfg.hidden_size, cfg.intermediate_size, case["tokens"]
    st["x"] = _randn(g, t, d)
    st["w"] = [_randn(g, e, d, f, std=0.02), _randn(g, e, d, f, std=0.02), _randn(g, e, f, d, std=0.02)]
    # routing of a trained gate: uneven over the experts, two distinct experts per token
    logits = _randn(g, t, e, dtype=torch.float32) + 0.5 * _randn(g, 1, e, dtype=torch.float32)
    top, st["idx"] = logits.softmax(-1).topk(cfg.num_experts_per_tok, dim=-1)
    st["idx"] = st["idx"].to(torch.int32)
    st["route"] = (top / top.sum(-1, keepdim=True)).to(BF16)
    for p in st["w"] + [st["route"]]:
      p.requires_grad_(True)
  elif kind in ("moe_train_fine", "moe_decode"):
    cfg = _config("deepseek-v2-lite")
    st["cfg"], st["layer"] = cfg, _init(_build(DeepseekV3MoE, cfg), g)
    st["x"] = _decided(_randn(g, case["batch"], case["seq"], cfg.hidden_size), st["layer"].gate.weight,
                       cfg.num_experts_per_tok)
  elif kind == "mla_train":
    cfg = _config("deepseek-v2-lite")
    st["cfg"], st["layer"] = cfg, _init(_build(DeepseekV3Attention, cfg), g)
    st["cos"], st["sin"] = _tables(case["seq"], _yarn_inv_freq(cfg))
    st["x"] = _randn(g, case["batch"], case["seq"], cfg.hidden_size)
  elif kind in ("decode", "prefill"):
    cfg = _config("deepseek-v2-lite", num_hidden_layers=ENGINE_LAYERS, first_k_dense_replace=ENGINE_LAYERS)
    model = _init(_build(DeepseekV3ForCausalLM, cfg), g)
    b = case["batch"]
    s = 1 if kind == "decode" else case["seq"]
    eng = DeepseekInferenceEngine(model, max_batch_size=b, max_seq_len=4096,
                                  attn_impl="absorb" if kind == "decode" else "naive")
    if kind == "decode":
      # what a prefill left in the cache: normalised latents and rotated keys
      for kv, pe in zip(eng.kv_cache, eng.pe_cache):
        kv[:, :case["start"]].normal_(0.0, 1.0, generator=g)
        pe[:, :case["start"]].normal_(0.0, 1.0, generator=g)
    st.update(cfg=cfg, model=model, engine=eng, start=case.get("start", 0),
              tokens=torch.randint(0, cfg.vocab_size, (b, s), device="cuda", generator=g))
  else:
    st["x"] = _randn(g, case["tokens"], case["dim"])
    st["layer"] = _init(_build(LlamaRMSNorm, case["dim"], 1e-5), g)
    st["dres"] = _randn(g, case["tokens"], case["dim"])
  if kind.endswith(("train", "wide", "fine")):
    st["x"].requires_grad_(True)
    st.setdefault("dy", _randn(g, *st["x"].shape))
  return st


# ------------------------------------------------------------------------------- one pass
def _parameters(st):
  if "layer" in st:
    return dict(st["layer"].named_parameters())
  if "w" in st:
    return {"w1": st["w"][0], "w3": st["w"][1], "w2": st["w"][2], "route": st["route"]}
  return {}


def run(st):
  kind = st["kind"]
  if kind in ("decode", "prefill"):
    return st["engine"].forward(st["tokens"], st["start"])
  if kind == "layer_eval":
    with torch.no_grad():
      return st["layer"](st["x"], st["cos"], st["sin"])
  if kind == "moe_decode":
    with torch.no_grad():
      return st["layer"](st["x"])
  params = _parameters(st)
  for p in [st["x"], *params.values()]:
    p.grad = None
  if kind == "layer_train" or kind == "mla_train":
    y = st["layer"](st["x"], st["cos"], st["sin"])
    y.backward(st["dy"])
  elif kind == "attn_train":
    y = ops.attention_qkv(st["x"], st["h"], st["hkv"], 128, causal=True, q_segment_ids=st["seg"])
    y.backward(st["dy"])
  elif kind == "head_train":
    _, y = st["layer"](st["x"], st["targets"], want_logits=False)
    y.backward()
  elif kind == "moe_train_wide":
    y = moe_ops.grouped_mlp(st["x"], st["route"], st["idx"], st["w"][0], st["w"][1], st["w"][2])
    y.backward(st["dy"])
  elif kind == "moe_train_fine":
    y = st["layer"](st["x"])
    y.backward(st["dy"])
  else:
    y, res = st["layer"].with_residual(st["x"])
    torch.autograd.backward([y, res], [st["dy"], st["dres"]])
  return {"y": y.detach(), "dx": st["x"].grad, **{f"d_{n}": p.grad for n, p in params.items()}}


# ------------------------------------------------------------------------------- what a pass needs
def work(case):
  kind = case["kind"]
  b, s = case.get("batch", 1), case.get("seq", 1)
  t = case.get("tokens", b * s)
  if kind in ("layer_eval", "layer_train"):
    w, d = (6144 + 4096) * 4096 + 3 * 4096 * 14336, 4096
    attn = 4 * b * 32 * 128 * s * (s + 1) / 2
    if kind == "layer_eval":
      return {"bytes": 2 * w + 4 * t * d, "flops": 2 * t * w + attn}
    return {"bytes": 4 * w + 8 * t * d, "flops": 6 * t * w + 3.5 * attn}
  if kind == "attn_train":
    h, hkv = case["heads"], case["kv_heads"]
    # packed segments of equal expected length halve the pairs again; count the plain causal ones
    # divided by the number of segments
    pairs = b * s * (s + 1) / 2 / max(1, case["segments"])
    return {"bytes": 2 * t * 128 * (2 * (h + 2 * hkv) + 2 * h), "flops": 14 * h * 128 * pairs}
  if kind == "head_train":
    d, v = 4096, 128256
    return {"bytes": 4 * d * v + 4 * t * d + 8 * t, "flops": 6 * t * d * v}
  if kind == "moe_train_wide":
    e, d, f, k = 8, 4096, 14336, 2
    hit = min(e, t * k)
    return {"bytes": 2 * hit * 3 * d * f + 2 * e * 3 * d * f + 8 * t * d, "flops": 6 * t * k * 3 * d * f}
  if kind in ("moe_train_fine", "moe_decode"):
    e, d, f, k = 64, 2048, 1408, 6
    hit = e * (1 - (1 - k / e) ** t)
    routed, shared = 3 * d * f, 3 * d * 2 * f
    if kind == "moe_decode":
      return {"bytes": 2 * (hit * routed + shared + e * d) + 4 * t * d, "flops": 2 * t * (k * routed + shared + e * d)}
    return {"bytes": 2 * (hit * routed + shared + e * d) + 2 * (e * routed + shared + e * d) + 8 * t * d,
            "flops": 6 * t * (k * routed + shared + e * d)}
  d, h, dn, dr, dv, c = 2048, 16, 128, 64, 128, 512
  proj = d * h * (dn + dr) + d * (c + dr) + c * h * (dn + dv) + h * dv * d
  if kind == "mla_train":
    attn = 2 * b * h * (dn + dr + dv) * s * (s + 1) / 2
    return {"bytes": 4 * proj + 8 * t * d, "flops": 6 * t * proj + 3.5 * attn}
  if kind in ("decode", "prefill"):
    mlp, vocab, n = 3 * d * 10944, 102400, ENGINE_LAYERS
    weights = 2 * (n * (proj + mlp) + vocab * d)
    if kind == "prefill":
      attn = n * 2 * b * h * (dn + dr + dv) * s * (s + 1) / 2
      cache = 2 * n * t * h * (dn + dr + dv)
      return {"bytes": weights + cache + 2 * t * d + 4 * b * vocab,
              "flops": 2 * t * n * (proj + mlp) + attn + 2 * b * vocab * d}
    keys = b * (case["start"] + 1)
    return {"bytes": weights + 2 * n * keys * (c + dr) + 2 * b * d + 4 * b * vocab,
            "flops": 2 * b * (n * (proj + mlp) + vocab * d) + n * 2 * keys * h * (2 * c + dr)}
  d = case["dim"]
  return {"bytes": 2 * t * d * 5, "flops": 12 * t * d}   # x, dy, dres in; y, dx out


# Largest relative error of an output that bf16 inputs, results and intermediates with fp32 sums give:
# four times the distance from exact() that was measured on a B200, 0.03 at most.
TOLERANCE = {
  "layer_eval": 0.025, "layer_train": 0.03, "attn_train": 0.012, "head_train": 0.012, "moe_train_wide": 0.018,
  "moe_train_fine": 0.016, "moe_decode": 0.01, "mla_train": 0.024, "decode": 0.03, "prefill": 0.03,
  "norm_train": 0.01,
}


def tolerance(case):
  return {"rel": TOLERANCE[case["kind"]], "max": 0.9}


# ------------------------------------------------------------------------------- 64-bit restatements
def _norm64(x, w, eps):
  return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate64(x, cos, sin, interleaved=False):
  """x [..., S, heads, D]; cos, sin [S, D/2] (a pair is (i, i + D/2), or (2i, 2i + 1) if interleaved, and stays there)."""
  half = x.shape[-1] // 2
  a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :half], x[..., half:])
  c, s = cos[:, None, :], sin[:, None, :]
  out = [a * c - b * s, b * c + a * s]
  return torch.stack(out, dim=-1).flatten(-2) if interleaved else torch.cat(out, dim=-1)


class _Attention64(torch.autograd.Function):
  """softmax(q k^T scale + mask) v, [B, S, H, D], one head at a time in both directions."""

  @staticmethod
  def _probs(q, k, scale, keep):
    return (q @ k.t() * scale).masked_fill_(~keep, float("-inf")).softmax(-1)

  @staticmethod
  def forward(ctx, q, k, v, scale, seg):
    ctx.save_for_backward(q, k, v, seg)
    ctx.scale = scale
    o = q.new_empty(*q.shape[:3], v.shape[-1])
    for b, h, kh, keep in _Attention64._heads(q, k, seg):
      o[b, :, h] = _Attention64._probs(q[b, :, h], k[b, :, kh], scale, keep) @ v[b, :, kh]
    return o

  @staticmethod
  def _heads(q, k, seg):
    causal = torch.ones(q.shape[1], k.shape[1], dtype=torch.bool, device=q.device).tril(k.shape[1] - q.shape[1])
    for b in range(q.shape[0]):
      keep = causal if seg is None else causal & (seg[b][:, None] == seg[b][None, :])
      for h in range(q.shape[2]):
        yield b, h, h * k.shape[2] // q.shape[2], keep

  @staticmethod
  def backward(ctx, do):
    q, k, v, seg = ctx.saved_tensors
    dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for b, h, kh, keep in _Attention64._heads(q, k, seg):
      p = _Attention64._probs(q[b, :, h], k[b, :, kh], ctx.scale, keep)
      dv[b, :, kh] += p.t() @ do[b, :, h]
      dp = do[b, :, h] @ v[b, :, kh].t()
      ds = p * (dp - (dp * p).sum(-1, keepdim=True)) * ctx.scale
      dq[b, :, h] = ds @ k[b, :, kh]
      dk[b, :, kh] += ds.t() @ q[b, :, h]
    return dq, dk, dv, None, None


def _experts64(x, w, idx, gate, up, down):
  """Sum over the selected experts; gate / up [E, D, F], down [E, F, D]."""
  y = torch.zeros_like(x)
  for e in range(gate.shape[0]):
    tok, slot = torch.nonzero(idx == e, as_tuple=True)
    if tok.numel():
      h = F.silu(x[tok] @ gate[e]) * (x[tok] @ up[e])
      y = y.index_add(0, tok, (h @ down[e]) * w[tok, slot][:, None])
  return y


def _moe64(x, p, cfg):
  flat = x.reshape(-1, x.shape[-1])
  scores = torch.sigmoid(flat @ p["gate.weight"].t())
  idx = scores.topk(cfg.num_experts_per_tok, dim=-1)[1]
  w = scores.gather(1, idx)
  w = w / w.sum(-1, keepdim=True) * float(cfg.routed_scaling_factor)
  y = _experts64(flat, w, idx, p["grouped.W_gate"], p["grouped.W_up"], p["grouped.W_down"])
  return y.view_as(x) + _mlp64(x, p, "shared_experts.")


def _mlp64(x, p, at):
  h = F.silu(x @ p[at + "gate_proj.weight"].t()) * (x @ p[at + "up_proj.weight"].t())
  return h @ p[at + "down_proj.weight"].t()


def _llama64(x, p, cfg, cos, sin):
  b, s, _ = x.shape
  h = _norm64(x, p["input_layernorm.weight"], cfg.rms_norm_eps)
  q, k, v = (
    (h @ p[f"self_attn.{n}_proj.weight"].t()).view(b, s, -1, 128) for n in ("q", "k", "v"))
  o = _Attention64.apply(_rotate64(q, cos, sin), _rotate64(k, cos, sin), v, 128 ** -0.5, None)
  x = x + o.reshape(b, s, -1) @ p["self_attn.o_proj.weight"].t()
  return x + _mlp64(_norm64(x, p["post_attention_layernorm.weight"], cfg.rms_norm_eps), p, "mlp.")


def _mla64(x, p, at, cfg, cos, sin, latents=None, rotated=None):
  """Latent attention; ``latents`` / ``rotated``: cached entries in front of x's own."""
  b, s, _ = x.shape
  h, dn, dr, dv, c = (cfg.num_attention_heads, cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim,
                      cfg.kv_lora_rank)
  m = 0.1 * cfg.rope_scaling["mscale_all_dim"] * math.log(cfg.rope_scaling["factor"]) + 1.0
  q = (x @ p[at + "q_proj.weight"].t()).view(b, s, h, dn + dr)
  q = torch.cat([q[..., :dn], _rotate64(q[..., dn:], cos, sin, True)], -1)
  kv = x @ p[at + "kv_a_proj_with_mqa.weight"].t()
  lat = _norm64(kv[..., :c], p[at + "kv_a_layernorm.weight"], 1e-6)
  rot = _rotate64(kv[..., None, c:], cos, sin, True)
  if latents is not None:
    lat, rot = torch.cat([latents, lat], 1), torch.cat([rotated[:, :, None], rot], 1)
  full = (lat @ p[at + "kv_b_proj.weight"].t()).view(b, -1, h, dn + dv)
  k = torch.cat([full[..., :dn], rot.expand(-1, -1, h, -1)], -1)
  o = _Attention64.apply(q, k, full[..., dn:], (dn + dr) ** -0.5 * m * m, None)
  return o.reshape(b, s, -1) @ p[at + "o_proj.weight"].t()


def _engine64(st):
  cfg, p = st["cfg"], {n: t.detach().double() for n, t in st["model"].named_parameters()}
  tokens, start = st["tokens"], st["start"]
  ang = (start + torch.arange(tokens.shape[1], dtype=torch.float64))[:, None] * _yarn_inv_freq(cfg)[None]
  cos, sin = ang.cos().cuda(), ang.sin().cuda()
  x = p["model.embed_tokens.weight"][tokens]
  for i in range(cfg.num_hidden_layers):
    at = f"model.layers.{i}."
    cached = [None, None] if not start else [t[i][:, :start].double() for t in (st["engine"].kv_cache, st["engine"].pe_cache)]
    h = _norm64(x, p[at + "input_layernorm.weight"], cfg.rms_norm_eps)
    x = x + _mla64(h, p, at + "self_attn.", cfg, cos, sin, *cached)
    x = x + _mlp64(_norm64(x, p[at + "post_attention_layernorm.weight"], cfg.rms_norm_eps), p, at + "mlp.")
  return _norm64(x[:, -1], p["model.norm.weight"], cfg.rms_norm_eps) @ p["lm_head.weight"].t()


def exact(case, seed):
  st = prepare(case, seed)
  kind = st["kind"]
  if kind in ("decode", "prefill"):
    with torch.no_grad():
      return _engine64(st)
  p = {n: t.detach().double().requires_grad_(True) for n, t in _parameters(st).items()}
  x = st["x"].detach().double().requires_grad_(True)
  cos, sin = (st[k].double() if k in st else None for k in ("cos", "sin"))
  with torch.set_grad_enabled(st["x"].requires_grad):
    if kind in ("layer_eval", "layer_train"):
      y = _llama64(x, p, st["cfg"], cos, sin)
    elif kind == "attn_train":
      b, s, _ = x.shape
      h, hkv = st["h"], st["hkv"]
      q, k, v = x.view(b, s, -1, 128).split([h, hkv, hkv], dim=2)
      y = _Attention64.apply(q, k, v, 128 ** -0.5, st["seg"])
    elif kind == "head_train":
      h = _norm64(x, p["norm.weight"], 1e-5)
      y = F.cross_entropy((h @ p["lm_head.weight"].t())[0], st["targets"][0], ignore_index=-100)
    elif kind == "moe_train_wide":
      y = _experts64(x, p["route"], st["idx"], p["w1"], p["w3"], p["w2"])
    elif kind in ("moe_train_fine", "moe_decode"):
      y = _moe64(x, p, st["cfg"])
    elif kind == "mla_train":
      y = _mla64(x, p, "", st["cfg"], cos, sin)
    else:
      y = _norm64(x, p["weight"], 1e-5)
  if not st["x"].requires_grad:
    return y
  if kind == "head_train":
    y.backward()
  elif kind == "norm_train":
    torch.autograd.backward([y, x], [st["dy"].double(), st["dres"].double()])
  else:
    y.backward(st["dy"].double())
  return {"y": y.detach(), "dx": x.grad, **{f"d_{n}": t.grad for n, t in p.items()}}
