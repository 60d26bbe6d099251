"""RMSNorm over many rows (rows streamed through shared memory, forward and backward) against 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, want):
  return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("rows,dim", [(2048, 8), (2049, 264), (2047, 1024), (1024, 1032), (3000, 2048), (2300, 2056), (1023, 4096),
                                      (5000, 4096), (2048, 4104), (1777, 5120), (2100, 5128), (2500, 8192)])
def test_forward_and_backward(cuda_lib, rows, dim, residual):
  """Widths around the row's share of a lane or thread, rows around the numbers of warps and the rule's edges.  y and dx are
  rounded to bf16 twice at most (2^-9 each), dw and rstd are fp32."""
  from torchprime_b200.ops import kernels as k
  torch.manual_seed(rows + dim)
  x, dy, dres = (torch.randn(rows, dim, device="cuda").bfloat16() for _ in range(3))
  w = (1 + 0.1 * torch.randn(dim, device="cuda")).bfloat16()
  y, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  dx, dw = k.rmsnorm_bwd(dy, x, w, rstd, dres=dres if residual else None)
  again = k.rmsnorm_bwd(dy, x, w, rstd, dres=dres if residual else None)
  xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
  r = torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)
  want = xd * r * wd
  want.backward(dy.double())
  assert _rel(rstd, r[:, 0]) < 1e-6
  assert _rel(y, want) < 2 ** -8
  assert _rel(dx, xd.grad + dres.double() if residual else xd.grad) < 2 ** -8
  assert _rel(dw, wd.grad) < 1e-5
  if rows >= 1024:
    assert all(torch.equal(a, b) for a, b in zip((dx, dw), again))


def test_bad_values_stay_in_their_row(cuda_lib):
  from torchprime_b200.ops import kernels as k
  x = torch.randn(2100, 2048, device="cuda").bfloat16()
  x[7, 3], x[2099, 0] = float("nan"), float("inf")
  w = torch.ones(2048, device="cuda").bfloat16()
  y, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  dx, dw = k.rmsnorm_bwd(torch.randn_like(x), x, w, rstd)
  good = torch.ones(2100, dtype=torch.bool, device="cuda")
  good[7] = good[2099] = False
  for t in (y, dx):
    assert torch.isfinite(t[good]).all()
    assert torch.isnan(t[7]).all() and not torch.isfinite(t[2099]).all()
  assert torch.isnan(dw).all()


@pytest.mark.parametrize("rows", [100, 4000])
def test_weight_gradient_holds_no_scratch(cuda_lib, rows):
  """The gradient that is returned keeps its own dim values alive and no partial sums."""
  from torchprime_b200.ops import kernels as k
  x = torch.randn(rows, 1024, device="cuda").bfloat16()
  w = torch.ones(1024, device="cuda").bfloat16()
  _, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  _, dw = k.rmsnorm_bwd(torch.randn_like(x), x, w, rstd)
  assert dw.untyped_storage().nbytes() == 4 * 1024


@pytest.mark.parametrize("rows", [300, 2100])
def test_weight_gradient_is_added_to_what_is_there(cuda_lib, rows):
  """From as many rows on as a call without a sum to add to does, this one takes the streamed kernel, so that its sum is that
  one's bit for bit (fewer rows are added with atomics: fp32 sums in any order)."""
  from torchprime_b200.ops import kernels as k
  x, dy = (torch.randn(rows, 2048, device="cuda").bfloat16() for _ in range(2))
  w = torch.ones(2048, device="cuda").bfloat16()
  _, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  dx, dw = k.rmsnorm_bwd(dy, x, w, rstd)
  old = torch.randn(2048, device="cuda")
  into = old.clone()
  dx2, got = k.rmsnorm_bwd(dy, x, w, rstd, dw_f32=into)
  assert got.data_ptr() == into.data_ptr() and torch.equal(dx, dx2)
  if rows >= 1024:
    assert torch.equal(into, old + dw)
  else:
    assert _rel(into, (old + dw).double()) < 1e-6


@pytest.mark.parametrize("rows,dim", [(887, 5120), (888, 5120), (889, 4104), (1333, 8192), (4499, 4096), (4500, 4096), (4501, 3080),
                                      (2047, 3072), (2048, 3072), (2050, 2056), (5000, 6144), (2999, 768), (3000, 768), (3001, 8),
                                      (11999, 2048), (12000, 2048), (12001, 776)])
def test_forward_of_wide_and_of_many_rows(cuda_lib, rows, dim):
  """Both sides of every edge between the forms; a residual of zeros asks for the one of a CTA to a row."""
  from torchprime_b200.ops import kernels as k
  torch.manual_seed(dim)
  x = torch.randn(rows, dim, device="cuda").bfloat16()
  w = (1 + 0.1 * torch.randn(dim, device="cuda")).bfloat16()
  y, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  y2, rstd2, _ = k.rmsnorm_fwd(x, w, 1e-5, res=torch.zeros_like(x), want_h=True)
  r = torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5)
  assert _rel(rstd, r[:, 0]) < 1e-6 and _rel(y, x.double() * r * w.double()) < 2 ** -8
  assert torch.equal(y, y2) and torch.equal(rstd, rstd2)


@pytest.mark.parametrize("dim", [8, 2048, 2056, 4096, 4104])
def test_few_and_many_rows_of_a_cta_each_are_the_same(cuda_lib, dim):
  """The form that asks for the weight with the row and the one that asks behind its sum differ in nothing else."""
  from torchprime_b200.ops import kernels as k
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  x, res = (torch.randn(2 * sms + 1, dim, device="cuda").bfloat16() for _ in range(2))
  w = (1 + 0.1 * torch.randn(dim, device="cuda")).bfloat16()
  for r in (None, res):
    many = k.rmsnorm_fwd(x, w, 1e-5, res=r, want_h=True)
    few = k.rmsnorm_fwd(x[:-1], w, 1e-5, res=None if r is None else r[:-1], want_h=True)
    assert all(a is None or torch.equal(a[:-1], b) for a, b in zip(many, few))


@pytest.mark.parametrize("rows,dim,streamed", [(591, 8192, False), (592, 8192, True), (600, 4104, True), (1023, 4096, False), (1024, 4096, True),
                                               (700, 6144, True)])
def test_backward_of_few_wide_rows(cuda_lib, rows, dim, streamed):
  """The streamed form, whose partial sums take scratch, begins earlier for wide rows."""
  from torchprime_b200.ops import kernels as k
  assert (cuda_lib.tpb_rmsnorm_bwd_parts(rows, dim) > 0) == streamed
  test_forward_and_backward(cuda_lib, rows, dim, True)


@pytest.mark.parametrize("rows,dim", [(12001, 8), (3001, 264), (3100, 768), (12000, 1024), (12001, 2048), (2100, 2056), (2049, 3072), (5000, 4096),
                                      (900, 4104), (1500, 5120), (1000, 8192)])
def test_all_forms_give_the_same_bits(cuda_lib, rows, dim):
  """Streamed rows against a CTA to a row: the forward that a residual (of zeros) asks for and the backward of few rows."""
  from torchprime_b200.ops import kernels as k
  torch.manual_seed(dim)
  x, dy, dres = (torch.randn(rows, dim, device="cuda").bfloat16() for _ in range(3))
  w = (1 + 0.1 * torch.randn(dim, device="cuda")).bfloat16()
  y, rstd, _ = k.rmsnorm_fwd(x, w, 1e-5)
  y2, rstd2, _ = k.rmsnorm_fwd(x, w, 1e-5, res=torch.zeros_like(x), want_h=True)
  assert torch.equal(y, y2) and torch.equal(rstd, rstd2)
  # with a residual's gradient the forms round its sum differently in some columns above 2048 (csrc/elementwise.cu, norm_dx)
  for res in (None, dres) if dim <= 2048 or 4096 < dim <= 6144 else (None,):
    dx, _ = k.rmsnorm_bwd(dy, x, w, rstd, dres=res)
    for at in range(0, rows, 500):
      part, _ = k.rmsnorm_bwd(dy[at:at + 500], x[at:at + 500], w, rstd[at:at + 500], dres=None if res is None else res[at:at + 500])
      assert torch.equal(dx[at:at + 500], part)
