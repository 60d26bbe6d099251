"""Cached latent-attention decode step (csrc/mla_decode.cu) against the engine's matrix-product form."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from torchprime_b200.config import compose
from torchprime_b200.experimental.deepseek_inference.engine import DeepseekInferenceEngine
from torchprime_b200.models.deepseek_v3 import DeepseekV3ForCausalLM
from torchprime_b200.models.model_utils import set_default_dtype
from torchprime_b200.ops import functional as ops
from torchprime_b200.ops import mla_decode


def _engine(**changes):
  cfg = compose("default", ["model=deepseek-v2-lite"]).model
  cfg["num_hidden_layers"], cfg["first_k_dense_replace"] = 1, 1
  cfg["vocab_size"], cfg["hidden_size"], cfg["intermediate_size"] = 512, 256, 256
  for n, v in changes.items():
    cfg[n] = v
  torch.manual_seed(0)
  with set_default_dtype(torch.bfloat16), torch.device("cuda"):
    model = DeepseekV3ForCausalLM(cfg).to("cuda")
  return DeepseekInferenceEngine(model, max_batch_size=9, max_seq_len=4096, attn_impl="absorb")


@pytest.mark.parametrize("heads", [16, 5])
@pytest.mark.parametrize("b,start", [(1, 0), (2, 30), (3, 31), (1, 32), (9, 33), (4, 1500), (1, 4095)])
def test_step_equals_the_matrix_product_form(cuda_lib, heads, b, start):
  eng = _engine(num_attention_heads=heads, num_key_value_heads=heads)
  attn = eng.model.model.layers[0].self_attn
  eng.kv_cache[0].normal_()
  eng.pe_cache[0].normal_()
  x = torch.randn(b, 1, 256, device="cuda", dtype=torch.bfloat16)
  res = torch.zeros(b, 1, 256, device="cuda", dtype=torch.bfloat16)
  positions = lambda: torch.full((b,), start, dtype=torch.int32, device="cuda")  # noqa: E731
  kv0, pe0 = eng.kv_cache[0].clone(), eng.pe_cache[0].clone()
  with torch.no_grad():
    got = eng._attention(0, attn, x, start, res, positions)
    kv1, pe1 = eng.kv_cache[0].clone(), eng.pe_cache[0].clone()
    eng.kv_cache[0].copy_(kv0)
    eng.pe_cache[0].copy_(pe0)
    old, mla_decode.supported = mla_decode.supported, lambda *a: False
    try:
      want = eng._attention(0, attn, x, start, res, positions)
    finally:
      mla_decode.supported = old
  # the caches: same rows written, one bf16 rounding of difference at most (another order of the norm's sum)
  for new, ref_, before in ((kv1, eng.kv_cache[0], kv0), (pe1, eng.pe_cache[0], pe0)):
    same = torch.ones_like(new, dtype=torch.bool)
    same[:b, start] = False
    assert torch.equal(new[same], before[same])
    assert torch.allclose(new[:b, start].float(), ref_[:b, start].float(), rtol=2.0 ** -7, atol=1e-6)
  # both forms compute in fp32; o is rounded to bf16 before the output projection
  assert ((got.float() - want.float()).norm() / want.float().norm()).item() < 2.0 ** -7


@pytest.mark.parametrize("heads,b,start", [(16, 5, 31), (37, 2, 3000), (38, 2, 3000), (75, 1, 3000), (74, 1, 40)])
def test_step_whose_last_kernel_fills_the_machine(cuda_lib, heads, b, start):
  """Both forms of the merge kernel (its CTAs all at once or not, four to a head and sequence), more ranges than the one asks for ahead."""
  test_step_equals_the_matrix_product_form(cuda_lib, heads, b, start)


def test_other_layouts_keep_the_matrix_product_form(cuda_lib):
  eng = _engine()
  a = eng.model.model.layers[0].self_attn
  q = torch.randn(2, 1, 16 * 192, device="cuda", dtype=torch.bfloat16)
  ckv = torch.randn(2, 1, 576, device="cuda", dtype=torch.bfloat16)
  args = (a.kv_a_layernorm.weight, eng.kv_cache[0], eng.pe_cache[0], a.kv_b_proj.weight, 16, 128, 64, 128, 512)
  assert not mla_decode.supported(q, ckv, *args)                       # gradients are recorded
  with torch.no_grad():
    assert mla_decode.supported(q, ckv, *args)
    assert not mla_decode.supported(q.repeat(1, 2, 1), ckv.repeat(1, 2, 1), *args)
    assert not mla_decode.supported(q.float(), ckv, *args)
    assert not mla_decode.supported(q, torch.randn(2, 1, 600, device="cuda", dtype=torch.bfloat16)[..., :576], *args)
    with ops.backend("torch"):
      assert not mla_decode.supported(q, ckv, *args)


def test_values_wider_than_the_kernel_takes(cuda_lib):
  """Value heads of more than 4096 columns run as matrix products."""
  eng = _engine(num_attention_heads=1, num_key_value_heads=1, v_head_dim=4104)
  x = torch.randn(2, 1, 256, device="cuda", dtype=torch.bfloat16)
  with torch.no_grad():
    y = eng._attention(0, eng.model.model.layers[0].self_attn, x, 0, x, lambda: torch.zeros(2, dtype=torch.int32, device="cuda"))
  assert y.shape == x.shape and bool(torch.isfinite(y).all())


@pytest.mark.parametrize("heads,c,start", [(16, 512, 40), (17, 64, 100), (3, 192, 700), (32, 448, 64)])
def test_widths_and_precision_of_the_split(cuda_lib, heads, c, start):
  """Other latent widths and head counts, against 64 bits: what the bf16 result's rounding leaves, for scores of +-20."""
  torch.manual_seed(c)
  b, dn, dv, n = 2, 128, 128, start + 1
  q = torch.randn(b, 1, heads * (dn + 64), device="cuda", dtype=torch.bfloat16) * 3
  ckv = torch.randn(b, 1, c + 64, device="cuda", dtype=torch.bfloat16)
  nw = torch.ones(c, device="cuda", dtype=torch.bfloat16)
  cos, sin = torch.ones(4096, 32, device="cuda"), torch.zeros(4096, 32, device="cuda")
  kv = torch.randn(b, 1024, c, device="cuda", dtype=torch.bfloat16)
  pe = torch.randn(b, 1024, 64, device="cuda", dtype=torch.bfloat16)
  w = (torch.randn(heads * (dn + dv), c, device="cuda") / c ** 0.5).to(torch.bfloat16)
  with torch.no_grad():
    got = mla_decode.absorb_step(q.clone(), ckv, nw, 1e-6, cos, sin, start, kv, pe, w, heads, dn, dv, 0.1, True)
  wd = w.double().view(heads, dn + dv, c)
  qd = q.double().view(b, heads, dn + 64)
  s = (torch.einsum("bhd,hdc,btc->bht", qd[..., :dn], wd[:, :dn], kv[:, :n].double())
       + torch.einsum("bhr,btr->bht", qd[..., dn:], pe[:, :n].double())) * 0.1
  o = torch.einsum("bht,btc,hjc->bhj", s.softmax(-1), kv[:, :n].double(), wd[:, dn:]).reshape(b, 1, -1)
  assert bool(((got.double() - o).abs() <= 2.0 ** -8 * o.abs() + 2e-5 * o.abs().max()).all()), (got.double() - o).abs().max()
