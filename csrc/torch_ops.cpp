// The framework's hot operators as native torch functions: argument checks, allocation, launch and the autograd node.
//
// A kernel of this library runs for a few microseconds at decode and short-sequence sizes; issued from Python (checks,
// ctypes, and in training a Python autograd function entered from the engine's thread) a launch cost 13 to 50 us of host
// time, which was all of the time of such calls.  Every function here answers None for whatever it is not meant for
// (other devices or types, layouts that need a copy, tensor subclasses, gradients collected in `main_grad`, traces,
// forward-mode AD, functorch transforms, dispatch modes), and the Python definition, which takes everything, goes on.
// Both issue the same launches with the same arguments.

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <cmath>
#include <optional>

#include "tpb.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace {

std::atomic<long long> g_launches{0};
PyObject* g_check = nullptr;         // _lib.check: raises KernelError for a non-zero code
PyObject* g_late_wgrads = nullptr;   // functional._deliver_wgrads: weights that got a main_grad after their forward
PyObject* g_late_norm = nullptr;     // functional._norm_wgrad
PyObject* g_main_grad = nullptr;     // "main_grad"

void check(int rc, const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (rc == 0) return;
  g_launches.fetch_sub(1, std::memory_order_relaxed);   // (counted by _lib.check)
  py::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
  throw py::error_already_set();
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Nothing watches or rewrites the operators of this thread but reverse-mode autograd.
bool unobserved() {
  return !at::tracer::impl::is_dispatch_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !torch::autograd::ForwardADLevel::try_get_by_idx(0) &&
         !c10::impl::tls_local_dispatch_key_set().included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

constexpr c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                        c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched,
                                        c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                        c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});

bool plain(const Tensor& t, at::ScalarType type = at::kBFloat16) {
  return t.defined() && t.is_cuda() && t.scalar_type() == type && t.layout() == at::kStrided && !t.key_set().has_any(kWrapped);
}
bool plain_rows(const Tensor& t, at::ScalarType type = at::kBFloat16) {   // and contiguous, with something in it
  return plain(t, type) && t.dim() > 0 && t.is_contiguous() && t.numel() > 0;
}
bool aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
bool recording(const Tensor& t) { return t.requires_grad(); }
bool small(int64_t n) { return n <= 0x7fffffff; }

Tensor empty_like_type(const Tensor& t, at::IntArrayRef sizes, at::ScalarType type) {
  return at::empty(sizes, t.options().dtype(type).requires_grad(false));
}
Tensor empty_as(const Tensor& t, at::IntArrayRef sizes) { return empty_like_type(t, sizes, t.scalar_type()); }
const void* cptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
const int* iptr(const Tensor& t) { return static_cast<const int*>(cptr(t)); }

std::vector<int64_t> with_last(const Tensor& t, int64_t last) {
  auto s = t.sizes().vec();
  s.back() = last;
  return s;
}

// The Python object of a parameter has a `main_grad` of its own.
bool has_main_grad(PyObject* o) {
  PyObject** d = _PyObject_GetDictPtr(o);
  if (d == nullptr || *d == nullptr) return false;
  PyObject* v = PyDict_GetItemWithError(*d, g_main_grad);
  return v != nullptr && v != Py_None;
}
bool any_main_grad(const Tensor* w, int n) {
  py::gil_scoped_acquire gil;
  for (int i = 0; i < n; ++i) {
    py::object o = py::reinterpret_steal<py::object>(THPVariable_Wrap(w[i]));
    if (has_main_grad(o.ptr())) return true;
  }
  return false;
}

// A tensor argument that may be None; false: something else.
bool unpack(py::handle h, Tensor& t) {
  if (h.is_none()) return true;
  if (!THPVariable_Check(h.ptr())) return false;
  t = THPVariable_Unpack(h.ptr());
  return true;
}

// Options that are a Python number or None; false: something else that counts as one (the Python definition converts it).
bool whole(py::handle h, int64_t none, int64_t& out) {
  out = none;
  if (h.is_none()) return true;
  int over = 0;
  if (!PyLong_Check(h.ptr())) return false;
  out = PyLong_AsLongLongAndOverflow(h.ptr(), &over);
  return over == 0;
}
bool real(py::handle h, double none, double& out) {
  out = none;
  if (h.is_none()) return true;
  if (!PyFloat_Check(h.ptr()) && !PyLong_Check(h.ptr())) return false;
  out = PyFloat_AsDouble(h.ptr());
  if (out != -1.0 || !PyErr_Occurred()) return true;
  PyErr_Clear();      // an integer beyond a double's range
  return false;
}

// One to three 2-D weights of one width that follow one another in one storage.
struct Weights {
  Tensor t[3];
  int n = 0;
  int64_t rows = 0, k = 0;
  bool grads = false, collected = false;   // some require a gradient; some collect it in a main_grad

  bool add(PyObject* o) {
    if (n == 3 || !THPVariable_Check(o)) return false;
    const Tensor& w = THPVariable_Unpack(o);
    if (!plain_rows(w) || w.dim() != 2) return false;
    if (n == 0) {
      k = w.size(1);
    } else {
      const Tensor& p = t[n - 1];
      if (w.size(1) != k || w.const_data_ptr() != static_cast<const char*>(p.const_data_ptr()) + 2 * p.numel() ||
          w.storage().data() != p.storage().data())
        return false;
    }
    t[n++] = w;
    rows += w.size(0);
    grads = grads || recording(w);
    collected = collected || has_main_grad(o);
    return true;
  }
  bool read(py::handle h) {
    if (!PyList_Check(h.ptr()) && !PyTuple_Check(h.ptr())) return add(h.ptr());
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(h.ptr());
    for (Py_ssize_t i = 0; i < len; ++i)
      if (!add(PySequence_Fast_GET_ITEM(h.ptr(), i))) return false;
    return n > 0;
  }
};

void gemm(const Tensor& a, const Tensor& b, const Tensor& c, int64_t m, int64_t n, int64_t k, bool a_mn, bool b_mn, int epi,
          const Tensor& aux = Tensor(), const Tensor& c2 = Tensor()) {
  const int64_t n_out = epi == TPB_EPI_SWIGLU ? n / 2 : epi == TPB_EPI_SWIGLU_BWD ? 2 * n : n;
  check(tpb_gemm_bf16(cptr(a), cptr(b), mptr(c), (int)m, (int)n, (int)k, a_mn ? m : k, b_mn ? n : k, n_out, a_mn, b_mn, epi,
                      1.f, cptr(aux), aux.defined() ? aux.size(-1) : 0, mptr(c2), c2.defined() ? n : 0, 0, stream()),
        "gemm");
}

// Gradients of weights that lie back to back, as slices of one product dy^T x.
variable_list weight_grads(const Tensor* w, int n, const Tensor& dy, const Tensor& x, int64_t rows, int64_t n_out, int64_t k) {
  variable_list out(n);
  if (any_main_grad(w, n)) {
    py::gil_scoped_acquire gil;
    py::list ws;
    for (int i = 0; i < n; ++i) ws.append(py::reinterpret_steal<py::object>(THPVariable_Wrap(w[i])));
    py::object r = py::reinterpret_borrow<py::object>(g_late_wgrads)(ws, py::cast(dy.view({rows, n_out})), py::cast(x.view({rows, k})));
    for (int i = 0; i < n; ++i)
      if (!r[py::int_(i)].is_none()) out[i] = r[py::int_(i)].cast<Tensor>();
    return out;
  }
  Tensor dw = empty_as(dy, {n_out, k});
  gemm(dy, x, dw, n_out, k, rows, true, true, TPB_EPI_BF16);
  for (int64_t i = 0, r = 0; i < n; r += w[i++].size(0)) out[i] = n == 1 ? dw : dw.narrow(0, r, w[i].size(0));
  return out;
}

// ------------------------------------------------------------------------------------------- linear
struct LinearFn : Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& residual, const Tensor& w0, const OptTensor& w1,
                        const OptTensor& w2, int64_t n_out) {
    const int64_t k = w0.size(1);
    Tensor y = empty_as(x, with_last(x, n_out));
    gemm(x, w0, y, x.numel() / k, n_out, k, false, false, residual ? TPB_EPI_BF16_RES : TPB_EPI_BF16,
         residual ? *residual : Tensor());
    variable_list saved{x, w0};
    if (w1) saved.push_back(*w1);
    if (w2) saved.push_back(*w2);
    ctx->save_for_backward(saved);
    ctx->saved_data["res"] = residual.has_value();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], *w = &saved[1];
    const int nw = (int)saved.size() - 1;
    const bool res = ctx->saved_data["res"].toBool();
    const Tensor dy = grads[0].contiguous();
    TORCH_CHECK(plain(dy), "linear: gradient of an unexpected kind");
    const int64_t k = w[0].size(1), n_out = dy.size(-1), rows = x.numel() / k;
    const int at = res ? 2 : 1;    // edge of the first weight
    variable_list out(5);
    if (ctx->needs_input_grad(0)) {
      out[0] = empty_as(x, x.sizes());
      gemm(dy, w[0], out[0], rows, k, n_out, false, true, TPB_EPI_BF16);
    }
    if (res) out[1] = grads[0];
    bool wanted = false;
    for (int i = 0; i < nw; ++i) wanted = wanted || ctx->needs_input_grad(at + i);
    if (wanted) {
      const variable_list dw = weight_grads(w, nw, dy, x, rows, n_out, k);
      for (int i = 0; i < nw; ++i) out[2 + i] = dw[i];
    }
    out.push_back(Tensor());
    return out;
  }
};

py::object linear(py::handle x_, py::handle ws_, py::handle res_) {
  Tensor x, residual;
  Weights w;
  if (!unobserved() || !unpack(x_, x) || !unpack(res_, residual) || !plain_rows(x) || !w.read(ws_)) return py::none();
  if (x.size(-1) != w.k || w.k % 8 || w.rows % 8 || x.get_device() != w.t[0].get_device()) return py::none();
  const int64_t rows = x.numel() / w.k;
  if (!small(rows) || !small(w.rows)) return py::none();
  if (residual.defined() && (!plain_rows(residual) || residual.numel() != rows * w.rows || residual.get_device() != x.get_device() ||
                             residual.size(-1) != w.rows))
    return py::none();
  const bool rec = at::GradMode::is_enabled() && (recording(x) || w.grads || (residual.defined() && recording(residual)));
  if (rec && (w.collected || (residual.defined() && residual.dim() != x.dim()))) return py::none();
  Tensor y;
  {
    py::gil_scoped_release nogil;
    if (rec) {
      auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
      y = LinearFn::apply(x, opt(residual), w.t[0], opt(w.t[1]), opt(w.t[2]), w.rows);
    } else {
      y = empty_as(x, with_last(x, w.rows));
      gemm(x, w.t[0], y, rows, w.rows, w.k, false, false, residual.defined() ? TPB_EPI_BF16_RES : TPB_EPI_BF16, residual);
    }
  }
  return py::cast(y);
}

// Two projections of the same few rows in one launch, without a graph; see functional.linear_pair.
py::object linear_pair(py::handle x_, py::handle w1_, py::handle w2_) {
  Tensor x;
  Weights w1, w2;
  if (at::GradMode::is_enabled() || !unobserved() || !unpack(x_, x) || !plain_rows(x) || !w1.add(w1_.ptr()) || !w2.add(w2_.ptr()))
    return py::none();
  const int64_t k = w1.k, rows = x.numel() / x.size(-1);
  if (x.size(-1) != k || w2.k != k || !small(rows) || !small(w1.rows) || !small(w2.rows) || x.get_device() != w1.t[0].get_device() ||
      x.get_device() != w2.t[0].get_device() || !tpb_linear_pair_pays((int)rows, (int)w1.rows, (int)w2.rows, (int)k))
    return py::none();       // (ahead of the results' allocation: a prefill comes here once a layer)
  Tensor y1, y2;
  int rc;
  {
    py::gil_scoped_release nogil;
    y1 = empty_as(x, with_last(x, w1.rows));
    y2 = empty_as(x, with_last(x, w2.rows));
    rc = tpb_linear_pair_bf16(cptr(x), cptr(w1.t[0]), cptr(w2.t[0]), mptr(y1), mptr(y2), (int)rows, (int)w1.rows, (int)w2.rows, (int)k,
                              stream());
    if (rc != -2) check(rc, "linear_pair");
  }
  if (rc == -2) return py::none();
  return py::make_tuple(y1, y2);
}

// ------------------------------------------------------------------------------------------- gate / up with SwiGLU
struct LinearSwigluFn : Function<LinearSwigluFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& wg, const Tensor& wu) {
    const int64_t k = wg.size(1), f = wg.size(0), rows = x.numel() / k;
    Tensor gu = empty_as(x, {rows, 2 * f}), act = empty_as(x, with_last(x, f));
    gemm(x, wg, act, rows, 2 * f, k, false, false, TPB_EPI_SWIGLU, Tensor(), gu);
    ctx->save_for_backward({x, gu, wg, wu});
    return act;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &gu = saved[1], *w = &saved[2];
    const int64_t k = w[0].size(1), f = w[0].size(0), rows = gu.size(0);
    const Tensor dact = grads[0].contiguous();
    TORCH_CHECK(plain(dact), "linear_swiglu: gradient of an unexpected kind");
    Tensor dgu = empty_as(gu, gu.sizes());
    check(tpb_swiglu_bwd(cptr(dact), cptr(gu), mptr(dgu), (int)rows, (int)f, stream()), "swiglu_bwd");
    variable_list out(3);
    if (ctx->needs_input_grad(0)) {
      out[0] = empty_as(x, x.sizes());
      gemm(dgu, w[0], out[0], rows, k, 2 * f, false, true, TPB_EPI_BF16);
    }
    if (ctx->needs_input_grad(1) || ctx->needs_input_grad(2)) {
      const variable_list dw = weight_grads(w, 2, dgu, x, rows, 2 * f, k);
      out[1] = dw[0];
      out[2] = dw[1];
    }
    return out;
  }
};

py::object linear_swiglu(py::handle x_, py::handle gate_, py::handle up_) {
  Tensor x;
  Weights w;
  if (!unobserved() || !unpack(x_, x) || !plain_rows(x) || !w.add(gate_.ptr()) || !w.add(up_.ptr())) return py::none();
  const int64_t f = w.t[0].size(0);
  if (w.t[1].size(0) != f || f % 8 || w.k % 8 || x.size(-1) != w.k || x.get_device() != w.t[0].get_device()) return py::none();
  const int64_t rows = x.numel() / w.k;
  if (!small(rows) || !small(2 * f)) return py::none();
  const bool rec = at::GradMode::is_enabled() && (recording(x) || w.grads);
  if (rec && w.collected) return py::none();
  Tensor y;
  {
    py::gil_scoped_release nogil;
    if (rec) {
      y = LinearSwigluFn::apply(x, w.t[0], w.t[1]);
    } else {
      y = empty_as(x, with_last(x, f));
      gemm(x, w.t[0], y, rows, 2 * f, w.k, false, false, TPB_EPI_SWIGLU);
    }
  }
  return py::cast(y);
}

// ------------------------------------------------------------------------------------------- the whole MLP
// y = (silu(x Wg^T) * (x Wu^T)) Wd^T (+ residual).  One node, so that the gradient of the activation needs no tensor: it
// becomes that of gate and up inside the down projection's input gradient, where that product is not a split one.
struct SwigluMlpFn : Function<SwigluMlpFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& residual, const Tensor& wg, const Tensor& wu,
                        const Tensor& wd) {
    const int64_t k = wg.size(1), f = wg.size(0), n = wd.size(0), rows = x.numel() / k;
    Tensor gu = empty_as(x, {rows, 2 * f}), act = empty_as(x, {rows, f}), y = empty_as(x, with_last(x, n));
    gemm(x, wg, act, rows, 2 * f, k, false, false, TPB_EPI_SWIGLU, Tensor(), gu);
    gemm(act, wd, y, rows, n, f, false, false, residual ? TPB_EPI_BF16_RES : TPB_EPI_BF16, residual ? *residual : Tensor());
    ctx->save_for_backward({x, gu, act, wg, wu, wd});
    ctx->saved_data["res"] = residual.has_value();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x = s[0], &gu = s[1], &act = s[2], *w = &s[3], &wd = s[5];
    const bool res = ctx->saved_data["res"].toBool();
    const Tensor dy = grads[0].contiguous();
    TORCH_CHECK(plain(dy), "swiglu_mlp: gradient of an unexpected kind");
    const int64_t k = w[0].size(1), f = w[0].size(0), n = wd.size(0), rows = gu.size(0);
    const int at = res ? 2 : 1;    // edge of the gate weight
    variable_list out(5);
    if (res) out[1] = grads[0];
    const bool up = ctx->needs_input_grad(at) || ctx->needs_input_grad(at + 1), in = ctx->needs_input_grad(0);
    if (in || up) {
      Tensor dgu = empty_as(gu, gu.sizes());
      if (tpb_gemm_swiglu_bwd_pays((int)rows, (int)f, (int)n)) {
        gemm(dy, wd, dgu, rows, f, n, false, true, TPB_EPI_SWIGLU_BWD, gu);
      } else {
        Tensor dact = empty_as(act, act.sizes());
        gemm(dy, wd, dact, rows, f, n, false, true, TPB_EPI_BF16);
        check(tpb_swiglu_bwd(cptr(dact), cptr(gu), mptr(dgu), (int)rows, (int)f, stream()), "swiglu_bwd");
      }
      if (in) {
        out[0] = empty_as(x, x.sizes());
        gemm(dgu, w[0], out[0], rows, k, 2 * f, false, true, TPB_EPI_BF16);
      }
      if (up) {
        const variable_list dw = weight_grads(w, 2, dgu, x, rows, 2 * f, k);
        out[2] = dw[0];
        out[3] = dw[1];
      }
    }
    if (ctx->needs_input_grad(at + 2)) out[4] = weight_grads(&wd, 1, dy, act, rows, n, f)[0];
    return out;
  }
};

py::object swiglu_mlp(py::handle x_, py::handle gate_, py::handle up_, py::handle down_, py::handle res_) {
  Tensor x, residual;
  Weights w, d;
  if (!unobserved() || !unpack(x_, x) || !unpack(res_, residual) || !plain_rows(x) || !w.add(gate_.ptr()) || !w.add(up_.ptr()) ||
      !d.add(down_.ptr()))
    return py::none();
  const int64_t f = w.t[0].size(0), n = d.rows, rows = x.numel() / x.size(-1);
  if (w.t[1].size(0) != f || d.k != f || f % 8 || w.k % 8 || n % 8 || x.size(-1) != w.k || !small(rows) || !small(2 * f) || !small(n) ||
      x.get_device() != w.t[0].get_device() || x.get_device() != d.t[0].get_device())
    return py::none();
  if (residual.defined() && (!plain_rows(residual) || residual.numel() != rows * n || residual.size(-1) != n ||
                             residual.get_device() != x.get_device()))
    return py::none();
  // (without gradients to record there is nothing to join)
  if (!(at::GradMode::is_enabled() && (recording(x) || w.grads || d.grads || (residual.defined() && recording(residual)))) ||
      w.collected || d.collected || (residual.defined() && residual.dim() != x.dim()))
    return py::none();
  Tensor y;
  {
    py::gil_scoped_release nogil;
    y = SwigluMlpFn::apply(x, residual.defined() ? OptTensor(residual) : OptTensor(), w.t[0], w.t[1], d.t[0]);
  }
  return py::cast(y);
}

// ------------------------------------------------------------------------------------------- norm
Tensor norm_fwd(const Tensor& x, const Tensor& w, double eps, const Tensor& rstd) {
  const int64_t d = x.size(-1);
  Tensor y = empty_as(x, x.sizes());
  check(tpb_rmsnorm_fwd(cptr(x), nullptr, cptr(w), mptr(y), nullptr, static_cast<float*>(mptr(rstd)), (int)(x.numel() / d),
                        (int)d, (float)eps, stream()),
        "rmsnorm_fwd");
  return y;
}

// dx (with the gradient of the residual branch added, if there is one) and dw.
variable_list norm_bwd(AutogradContext* ctx, const Tensor& dy_, const Tensor& dres_) {
  const variable_list saved = ctx->get_saved_variables();
  const Tensor &x = saved[0], &w = saved[1], &rstd = saved[2];
  const Tensor dy = dy_.contiguous(), dres = dres_.defined() ? dres_.contiguous() : Tensor();
  TORCH_CHECK(plain(dy) && (!dres.defined() || plain(dres)), "rms_norm: gradient of an unexpected kind");
  const int64_t d = x.size(-1);
  const int rows = (int)(x.numel() / d);
  const bool late = ctx->needs_input_grad(1) && any_main_grad(&w, 1);
  // fp32 sums and scratch in one allocation, unless the sums are handed on and would keep the scratch alive
  const int64_t n = tpb_rmsnorm_bwd_parts(rows, (int)d);
  Tensor dx = empty_as(x, x.sizes()), sums, parts, dw;
  if (late) {
    sums = empty_like_type(w, {d}, at::kFloat);
    if (n) parts = empty_like_type(w, {n, d}, at::kFloat);
  } else {
    sums = empty_like_type(w, {1 + n, d}, at::kFloat);
    if (ctx->needs_input_grad(1)) dw = empty_as(w, {d});
  }
  float* const sums_p = static_cast<float*>(mptr(sums));
  float* const parts_p = late ? static_cast<float*>(mptr(parts)) : n ? sums_p + d : nullptr;
  check(tpb_rmsnorm_bwd_dw(cptr(dy), cptr(x), cptr(w), static_cast<const float*>(cptr(rstd)), cptr(dres), mptr(dx),
                           sums_p, mptr(dw), parts_p, 0, rows, (int)d, stream()),
        "rmsnorm_bwd");
  if (late) {
    py::gil_scoped_acquire gil;
    py::reinterpret_borrow<py::object>(g_late_norm)(py::reinterpret_steal<py::object>(THPVariable_Wrap(w)), py::cast(sums));
  }
  return {dx, dw, Tensor()};
}

struct NormFn : Function<NormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    Tensor rstd = empty_like_type(x, {x.numel() / x.size(-1)}, at::kFloat);
    Tensor y = norm_fwd(x, w, eps, rstd);
    ctx->save_for_backward({x, w, rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return norm_bwd(ctx, grads[0], Tensor()); }
};

// (norm(x), x); see functional._RMSNormPassFn.
struct NormPassFn : Function<NormPassFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    Tensor rstd = empty_like_type(x, {x.numel() / x.size(-1)}, at::kFloat);
    Tensor y = norm_fwd(x, w, eps, rstd);
    ctx->save_for_backward({x, w, rstd});
    return {y, x.view_as(x)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return norm_bwd(ctx, grads[0], grads[1]); }
};

bool norm_args(py::handle x_, py::handle w_, Tensor& x, Tensor& w) {
  if (!unobserved() || !unpack(x_, x) || !plain_rows(x) || !THPVariable_Check(w_.ptr()) ||
      (at::GradMode::is_enabled() && has_main_grad(w_.ptr())))
    return false;
  w = THPVariable_Unpack(w_.ptr());
  const int64_t d = x.size(-1);
  return plain_rows(w) && w.dim() == 1 && w.numel() == d && d % 8 == 0 && d <= 8192 && small(x.numel() / d) &&
         w.get_device() == x.get_device();
}

py::object rms_norm(py::handle x_, py::handle w_, double eps) {
  Tensor x, w, y;
  if (!norm_args(x_, w_, x, w)) return py::none();
  {
    py::gil_scoped_release nogil;
    y = at::GradMode::is_enabled() && (recording(x) || recording(w)) ? NormFn::apply(x, w, eps) : norm_fwd(x, w, eps, Tensor());
  }
  return py::cast(y);
}

py::object rms_norm_residual(py::handle x_, py::handle w_, double eps) {
  Tensor x, w;
  if (!norm_args(x_, w_, x, w)) return py::none();
  variable_list y;
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && (recording(x) || recording(w))) y = NormPassFn::apply(x, w, eps);
    else y = {norm_fwd(x, w, eps, Tensor()), x.view_as(x)};
  }
  return py::make_tuple(y[0], y[1]);
}

// ------------------------------------------------------------------------------------------- rotary embedding, in place
void rope_launch(const Tensor& x, const Tensor& cos, const Tensor& sin, const Tensor& pos, int64_t heads, int64_t dim,
                 int64_t seq, bool interleaved, int64_t col0, int64_t head_stride, bool inverse) {
  const int64_t c = x.size(-1);
  check(tpb_rope_strided(mptr(x), c, (int)col0, (int)heads, (int)dim, (int)head_stride, static_cast<const float*>(cptr(cos)),
                         static_cast<const float*>(cptr(sin)), iptr(pos), (int)(x.numel() / c), (int)seq, inverse, interleaved,
                         stream()),
        "rope");
}

struct RopeFn : Function<RopeFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& cos, const Tensor& sin, const OptTensor& pos,
                        int64_t heads, int64_t dim, int64_t seq, bool interleaved, int64_t col0, int64_t head_stride) {
    rope_launch(x, cos, sin, pos ? *pos : Tensor(), heads, dim, seq, interleaved, col0, head_stride, false);
    ctx->mark_dirty({x});
    if (pos) ctx->save_for_backward({cos, sin, *pos}); else ctx->save_for_backward({cos, sin});
    ctx->saved_data["a"] = std::vector<int64_t>{heads, dim, seq, interleaved, col0, head_stride};
    return x;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const auto a = ctx->saved_data["a"].toIntVector();
    // (the gradient of a projection that was rotated in place has no other reader: it is rotated in place as well)
    Tensor d = grads[0].contiguous();
    TORCH_CHECK(plain(d), "rope: gradient of an unexpected kind");
    rope_launch(d, saved[0], saved[1], saved.size() > 2 ? saved[2] : Tensor(), a[0], a[1], a[2], a[3] != 0, a[4], a[5], true);
    variable_list out(10);
    out[0] = d;
    return out;
  }
};

py::object rope(py::handle x_, py::handle cos_, py::handle sin_, int64_t heads, int64_t dim, int64_t seq, py::handle pos_,
                bool interleaved, int64_t col0, py::handle head_stride_) {
  Tensor x, cos, sin, pos;
  if (!unobserved() || !unpack(x_, x) || !unpack(cos_, cos) || !unpack(sin_, sin) || !unpack(pos_, pos) || !plain_rows(x) ||
      !plain_rows(cos, at::kFloat) || !plain_rows(sin, at::kFloat) || recording(cos) || recording(sin))
    return py::none();
  const int64_t c = x.size(-1), tokens = x.numel() / c;
  int64_t hs;
  if (!whole(head_stride_, 0, hs)) return py::none();
  if (hs == 0) hs = dim;
  if (cos.size(-1) != dim / 2 || sin.size(-1) != dim / 2 || !small(tokens) || !small(c)) return py::none();
  if (pos.defined() && (!plain_rows(pos, at::kInt) || pos.numel() != tokens)) return py::none();
  const bool rec = at::GradMode::is_enabled() && recording(x);
  {
    py::gil_scoped_release nogil;
    if (rec) {
      x = RopeFn::apply(x, cos, sin, pos.defined() ? OptTensor(pos) : OptTensor(), heads, dim, seq, interleaved, col0, hs);
    } else {
      rope_launch(x, cos, sin, pos, heads, dim, seq, interleaved, col0, hs, false);
      if (!x.is_inference()) x.unsafeGetTensorImpl()->bump_version();   // an earlier graph that saved x has to notice
    }
  }
  if (!rec) return py::reinterpret_borrow<py::object>(x_);
  return py::cast(x);
}

// ------------------------------------------------------------------------------------------- attention
struct AttnShape {
  int64_t b, sq, sk, hq, hkv, dqk, dv, ldq, ldk, ldv;
  double scale;
  bool causal;
  int64_t window;
  double softcap;
};

// (smallest, largest) segment id of every 64 tokens, where the kernels use it; see attention_sm100._seg_ranges.
Tensor seg_table(const Tensor& seg, int64_t b, int64_t s) {
  Tensor t = empty_as(seg, {b, (s + 63) / 64, 2});
  check(tpb_attn_seg_ranges(iptr(seg), static_cast<int*>(mptr(t)), (int)b, (int)s, stream()), "attn_seg_ranges");
  return t;
}

void attn_fwd(const AttnShape& a, const void* q, const void* k, const void* v, const Tensor& o, const Tensor& lse,
              const Tensor& pos, const Tensor& q_seg, const Tensor& kv_seg, const Tensor& q_rng, const Tensor& kv_rng) {
  check(tpb_attn_fwd_softcap(q, k, v, mptr(o), static_cast<float*>(mptr(lse)), (int)a.b, (int)a.sq, (int)a.sk, (int)a.hq,
                             (int)a.hkv, (int)a.dqk, (int)a.dv, a.ldq, a.ldk, a.ldv, a.hq * a.dv, (float)a.scale, a.causal,
                             (int)a.window, iptr(pos), iptr(q_seg), iptr(kv_seg), iptr(q_rng), iptr(kv_rng), (float)a.softcap,
                             stream()),
        "attn_fwd");
}

void attn_bwd(const AttnShape& a, const Tensor& d_o, const void* q, const void* k, const void* v, const Tensor& o,
              const Tensor& lse, void* dq, void* dk, void* dv, int64_t lddq, int64_t lddk, int64_t lddv, const Tensor& pos,
              const Tensor& q_seg, const Tensor& kv_seg, const Tensor& q_rng, const Tensor& kv_rng) {
  Tensor scratch = empty_like_type(lse, {tpb_attn_bwd_scratch_floats((int)a.b, (int)a.sq, (int)a.hq)}, at::kFloat);
  check(tpb_attn_bwd_softcap(cptr(d_o), q, k, v, cptr(o), static_cast<const float*>(cptr(lse)),
                             static_cast<float*>(mptr(scratch)), dq, dk, dv, (int)a.b, (int)a.sq, (int)a.sk, (int)a.hq,
                             (int)a.hkv, (int)a.dqk, (int)a.dv, a.ldq, a.ldk, a.ldv, a.hq * a.dv, lddq, lddk, lddv,
                             (float)a.scale, a.causal, (int)a.window, iptr(pos), iptr(q_seg), iptr(kv_seg), iptr(q_rng),
                             iptr(kv_rng), (float)a.softcap, stream()),
        "attn_bwd");
}

// Ids or positions as the kernels read them: one contiguous int32 per token.
bool per_token(py::handle h, int64_t tokens, Tensor& out) {
  Tensor t;
  if (!unpack(h, t)) return false;
  if (!t.defined()) return true;
  if (!(plain(t, at::kInt) || plain(t, at::kLong)) || t.numel() != tokens) return false;
  out = t.reshape(-1).to(at::kInt).contiguous();
  return true;
}

OptTensor some(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
Tensor get(const OptTensor& t) { return t ? *t : Tensor(); }

AttnShape qkv_shape(const Tensor& qkv, int64_t hq, int64_t hkv, double scale, bool causal, int64_t window) {
  const int64_t w = qkv.size(2);
  return {qkv.size(0), qkv.size(1), qkv.size(1), hq, hkv, 128, 128, w, w, w, scale, causal, window, 0.0};
}

struct AttentionQKVFn : Function<AttentionQKVFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const OptTensor& pos_, const OptTensor& seg_, int64_t hq,
                        int64_t hkv, double scale, bool causal, int64_t window) {
    const AttnShape a = qkv_shape(qkv, hq, hkv, scale, causal, window);
    const Tensor pos = get(pos_), seg = get(seg_), rng = seg.defined() && a.sk > 256 ? seg_table(seg, a.b, a.sk) : Tensor();
    Tensor o = empty_as(qkv, {a.b, a.sq, hq, 128}), lse = empty_like_type(qkv, {a.b, hq, a.sq}, at::kFloat);
    const char* at0 = static_cast<const char*>(cptr(qkv));
    attn_fwd(a, at0, at0 + 2 * hq * 128, at0 + 2 * (hq + hkv) * 128, o, lse, pos, seg, seg, rng, rng);
    ctx->save_for_backward({qkv, o, lse, pos, seg, rng});
    ctx->saved_data["i"] = std::vector<int64_t>{hq, hkv, causal, window};
    ctx->saved_data["s"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor& qkv = s[0];
    const auto i = ctx->saved_data["i"].toIntVector();
    const AttnShape a = qkv_shape(qkv, i[0], i[1], ctx->saved_data["s"].toDouble(), i[2] != 0, i[3]);
    const Tensor d_o = grads[0].contiguous();
    TORCH_CHECK(plain(d_o), "attention: gradient of an unexpected kind");
    Tensor buf = empty_as(qkv, qkv.sizes());
    const char* x = static_cast<const char*>(cptr(qkv));
    char* d = static_cast<char*>(mptr(buf));
    const int64_t ko = 2 * a.hq * 128, vo = 2 * (a.hq + a.hkv) * 128;
    attn_bwd(a, d_o, x, x + ko, x + vo, s[1], s[2], d, d + ko, d + vo, a.ldq, a.ldq, a.ldq, s[3], s[4], s[4], s[5], s[5]);
    variable_list out(8);
    out[0] = buf;
    return out;
  }
};

py::object attention_qkv(py::handle x_, int64_t hq, int64_t hkv, int64_t d, bool causal, py::handle scale_, py::handle window_,
                         py::handle seg_, py::handle pos_) {
  Tensor x, seg, pos, o;
  if (!unobserved() || !unpack(x_, x) || !plain_rows(x) || x.dim() != 3 || d != 128 || hq <= 0 || hkv <= 0 || hq % hkv ||
      x.size(2) != (hq + 2 * hkv) * d || !small(x.size(0) * x.size(1)))
    return py::none();
  if (!per_token(seg_, x.size(0) * x.size(1), seg) || !per_token(pos_, x.size(0) * x.size(1), pos)) return py::none();
  double scale;
  int64_t window;
  if (!real(scale_, 1.0 / std::sqrt((double)d), scale) || !whole(window_, 0, window)) return py::none();
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && recording(x)) {
      o = AttentionQKVFn::apply(x, some(pos), some(seg), hq, hkv, scale, causal, window);
    } else {
      const AttnShape a = qkv_shape(x, hq, hkv, scale, causal, window);
      const Tensor rng = seg.defined() && a.sk > 256 ? seg_table(seg, a.b, a.sk) : Tensor();
      Tensor lse = empty_like_type(x, {a.b, hq, a.sq}, at::kFloat);
      o = empty_as(x, {a.b, a.sq, hq, 128});
      const char* at0 = static_cast<const char*>(cptr(x));
      attn_fwd(a, at0, at0 + 2 * hq * 128, at0 + 2 * (hq + hkv) * 128, o, lse, pos, seg, seg, rng, rng);
    }
  }
  return py::cast(o);
}

AttnShape separate_shape(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool causal, int64_t window,
                         double softcap) {
  return {q.size(0), q.size(1), k.size(1), q.size(2), k.size(2), q.size(3), v.size(3), q.stride(1), k.stride(1), v.stride(1),
          scale, causal, window, softcap};
}

struct AttentionFn : Function<AttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& pos_,
                        const OptTensor& q_seg_, const OptTensor& kv_seg_, double scale, bool causal, int64_t window,
                        double softcap) {
    const AttnShape a = separate_shape(q, k, v, scale, causal, window, softcap);
    const Tensor pos = get(pos_), q_seg = get(q_seg_), kv_seg = get(kv_seg_);
    Tensor q_rng, kv_rng;
    if (q_seg.defined() && kv_seg.defined() && a.sk > 256) {
      kv_rng = seg_table(kv_seg, a.b, a.sk);
      q_rng = a.sq == a.sk && cptr(q_seg) == cptr(kv_seg) ? kv_rng : seg_table(q_seg, a.b, a.sq);
    }
    Tensor o = empty_as(q, {a.b, a.sq, a.hq, a.dv}), lse = empty_like_type(q, {a.b, a.hq, a.sq}, at::kFloat);
    attn_fwd(a, cptr(q), cptr(k), cptr(v), o, lse, pos, q_seg, kv_seg, q_rng, kv_rng);
    ctx->save_for_backward({q, k, v, o, lse, pos, q_seg, kv_seg, q_rng, kv_rng});
    ctx->saved_data["i"] = std::vector<int64_t>{causal, window};
    ctx->saved_data["s"] = std::vector<double>{scale, softcap};
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list t = ctx->get_saved_variables();
    const Tensor &q = t[0], &k = t[1], &v = t[2];
    const auto i = ctx->saved_data["i"].toIntVector();
    const auto s = ctx->saved_data["s"].toDoubleVector();
    const AttnShape a = separate_shape(q, k, v, s[0], i[0] != 0, i[1], s[1]);
    const Tensor d_o = grads[0].contiguous();
    TORCH_CHECK(plain(d_o), "attention: gradient of an unexpected kind");
    Tensor dq = empty_as(q, q.sizes()), dk = empty_as(k, k.sizes()), dv = empty_as(v, v.sizes());
    attn_bwd(a, d_o, cptr(q), cptr(k), cptr(v), t[3], t[4], mptr(dq), mptr(dk), mptr(dv), a.hq * a.dqk, a.hkv * a.dqk,
             a.hkv * a.dv, t[5], t[6], t[7], t[8], t[9]);
    variable_list out(10);
    out[0] = dq; out[1] = dk; out[2] = dv;
    return out;
  }
};

// [B, S, H, D] with unit stride over D, D over heads, one pitch per token, batches back to back.
bool token_major(const Tensor& t) {
  return plain(t) && t.dim() == 4 && t.numel() > 0 && t.stride(3) == 1 && t.stride(2) == t.size(3) && t.stride(1) % 8 == 0 &&
         (t.size(0) == 1 || t.stride(0) == t.size(1) * t.stride(1)) && aligned(t);
}
// Three slices of one projection, whose gradients the Python definition lays out as one.
bool one_storage(const Tensor& q, const Tensor& k, const Tensor& v) {
  return q.storage().data() == k.storage().data() || q.storage().data() == v.storage().data();
}

py::object attention(py::handle q_, py::handle k_, py::handle v_, bool causal, py::handle scale_, py::handle window_,
                     py::handle qseg_, py::handle kvseg_, py::handle softcap_, py::handle pos_, int64_t max_wide_queries) {
  Tensor q, k, v, q_seg, kv_seg, pos, o;
  if (!unobserved() || !unpack(q_, q) || !unpack(k_, k) || !unpack(v_, v) || !token_major(q) || !token_major(k) || !token_major(v))
    return py::none();
  const int64_t b = q.size(0), sq = q.size(1), sk = k.size(1), dqk = q.size(3);
  double softcap, scale;
  int64_t window;
  if (!real(softcap_, 0.0, softcap) || !real(scale_, 1.0 / std::sqrt((double)dqk), scale) || !whole(window_, 0, window))
    return py::none();
  if (k.size(0) != b || v.size(0) != b || v.size(1) != sk || k.size(3) != dqk || v.size(3) != 128 || (dqk != 128 && dqk != 192) ||
      k.size(2) != v.size(2) || q.size(2) % k.size(2) || softcap < 0 || (softcap > 0 && dqk != 128) || one_storage(q, k, v) ||
      (dqk != 128 && sq > max_wide_queries) || !small(b * sq) || !small(b * sk))
    return py::none();
  if (!per_token(qseg_, b * sq, q_seg) || !per_token(pos_, b * sq, pos)) return py::none();
  if (kvseg_.is_none()) {
    if (q_seg.defined() && sq != sk) return py::none();
    kv_seg = q_seg;
  } else if (!per_token(kvseg_, b * sk, kv_seg)) {
    return py::none();
  }
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && (recording(q) || recording(k) || recording(v))) {
      o = AttentionFn::apply(q, k, v, some(pos), some(q_seg), some(kv_seg), scale, causal, window, softcap);
    } else {
      const AttnShape a = separate_shape(q, k, v, scale, causal, window, softcap);
      Tensor q_rng, kv_rng;
      if (q_seg.defined() && kv_seg.defined() && sk > 256) {
        kv_rng = seg_table(kv_seg, b, sk);
        q_rng = sq == sk && cptr(q_seg) == cptr(kv_seg) ? kv_rng : seg_table(q_seg, b, sq);
      }
      Tensor lse = empty_like_type(q, {b, a.hq, sq}, at::kFloat);
      o = empty_as(q, {b, sq, a.hq, a.dv});
      attn_fwd(a, cptr(q), cptr(k), cptr(v), o, lse, pos, q_seg, kv_seg, q_rng, kv_rng);
    }
  }
  return py::cast(o);
}

// ------------------------------------------------------------------------------------------- latent attention layout
struct LatentSplitFn : Function<LatentSplitFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& ckv, int64_t c) {
    return {ckv.narrow(-1, 0, c).contiguous(), ckv.narrow(-1, c, ckv.size(-1) - c).contiguous()};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) { return {at::cat({g[0], g[1]}, -1), Tensor()}; }
};

py::object latent_split(py::handle x_, int64_t c) {
  Tensor x;
  if (!unobserved() || !unpack(x_, x) || !plain_rows(x) || c <= 0 || c >= x.size(-1)) return py::none();
  variable_list y;
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && recording(x)) y = LatentSplitFn::apply(x, c);
    else y = {x.narrow(-1, 0, c).contiguous(), x.narrow(-1, c, x.size(-1) - c).contiguous()};
  }
  return py::make_tuple(y[0], y[1]);
}

// The same with the rotary key rotated on the way (functional.latent_split_rope).
variable_list latent_rope_now(const Tensor& x, const Tensor& cos, const Tensor& sin, const Tensor& pos, int64_t c, int64_t seq,
                              bool interleaved) {
  const int64_t dr = x.size(-1) - c;
  Tensor lat = empty_as(x, with_last(x, c)), rot = empty_as(x, with_last(x, dr));
  check(tpb_latent_split(cptr(x), mptr(lat), mptr(rot), static_cast<const float*>(cptr(cos)), static_cast<const float*>(cptr(sin)),
                         iptr(pos), x.numel() / x.size(-1), (int)seq, (int)c, (int)dr, interleaved, stream()),
        "latent_split");
  return {lat, rot};
}

struct LatentRopeFn : Function<LatentRopeFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& cos, const Tensor& sin, const OptTensor& pos,
                               int64_t c, int64_t seq, bool interleaved) {
    ctx->save_for_backward({cos, sin, get(pos)});
    ctx->saved_data["a"] = std::vector<int64_t>{seq, interleaved};
    return latent_rope_now(x, cos, sin, get(pos), c, seq, interleaved);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const auto a = ctx->saved_data["a"].toIntVector();
    const Tensor dlat = g[0].contiguous(), drot = g[1].contiguous();
    TORCH_CHECK(plain(dlat) && plain(drot), "latent_split: gradient of an unexpected kind");
    const int64_t c = dlat.size(-1), dr = drot.size(-1);
    Tensor dx = empty_as(dlat, with_last(dlat, c + dr));
    check(tpb_latent_join(cptr(dlat), cptr(drot), mptr(dx), static_cast<const float*>(cptr(s[0])),
                          static_cast<const float*>(cptr(s[1])), iptr(s[2]), dlat.numel() / c, (int)a[0], (int)c, (int)dr, a[1] != 0,
                          stream()),
          "latent_join");
    variable_list out(7);
    out[0] = dx;
    return out;
  }
};

py::object latent_split_rope(py::handle x_, int64_t c, py::handle cos_, py::handle sin_, int64_t seq, py::handle pos_,
                             bool interleaved) {
  Tensor x, cos, sin, pos;
  if (!unobserved() || !unpack(x_, x) || !unpack(cos_, cos) || !unpack(sin_, sin) || !unpack(pos_, pos) || !plain_rows(x) ||
      !plain_rows(cos, at::kFloat) || !plain_rows(sin, at::kFloat) || recording(cos) || recording(sin) || !aligned(x))
    return py::none();
  const int64_t dr = x.size(-1) - c, tokens = x.numel() / x.size(-1);
  if (c < 8 || c % 8 || dr < 16 || dr % 16 || cos.size(-1) != dr / 2 || sin.size(-1) != dr / 2 || seq < 1 || !small(tokens) ||
      (pos.defined() && (!plain_rows(pos, at::kInt) || pos.numel() != tokens)))
    return py::none();
  variable_list y;
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && recording(x)) y = LatentRopeFn::apply(x, cos, sin, some(pos), c, seq, interleaved);
    else y = latent_rope_now(x, cos, sin, pos, c, seq, interleaved);
  }
  return py::make_tuple(y[0], y[1]);
}

variable_list mla_pack_now(const Tensor& kv, const Tensor& rot, int64_t heads, int64_t dn, int64_t dv) {
  const int64_t b = rot.size(0), s = rot.size(1), dr = rot.size(2);
  Tensor k = empty_as(kv, {b, s, heads, dn + dr}), v = empty_as(kv, {b, s, heads, dv});
  check(tpb_mla_pack(cptr(kv), cptr(rot), dr, mptr(k), mptr(v), b * s, (int)heads, (int)dn, (int)dr, (int)dv, stream()),
        "mla_pack");
  return {k, v};
}

struct MlaPackFn : Function<MlaPackFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& kv, const Tensor& rot, int64_t heads, int64_t dn, int64_t dv) {
    ctx->saved_data["i"] = std::vector<int64_t>{heads, dn, dv};
    return mla_pack_now(kv, rot, heads, dn, dv);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto i = ctx->saved_data["i"].toIntVector();
    const int64_t heads = i[0], dn = i[1], dv = i[2];
    const Tensor dk = g[0].contiguous(), dvv = g[1].contiguous();
    TORCH_CHECK(plain(dk) && plain(dvv), "mla_pack: gradient of an unexpected kind");
    const int64_t b = dk.size(0), s = dk.size(1), dr = dk.size(3) - dn;
    Tensor dkv = empty_as(dk, {b, s, heads * (dn + dv)}), drot = empty_as(dk, {b, s, dr});
    check(tpb_mla_unpack(cptr(dk), cptr(dvv), mptr(dkv), mptr(drot), b * s, (int)heads, (int)dn, (int)dr, (int)dv, stream()),
          "mla_unpack");
    return {dkv, drot, Tensor(), Tensor(), Tensor()};
  }
};

py::object mla_pack(py::handle kv_, py::handle rot_, int64_t heads, int64_t dn, int64_t dv) {
  Tensor kv, rot;
  if (!unobserved() || !unpack(kv_, kv) || !unpack(rot_, rot) || !plain_rows(kv) || !plain_rows(rot) || rot.dim() != 3 ||
      kv.dim() != 3 || kv.size(0) != rot.size(0) || kv.size(1) != rot.size(1) || kv.size(2) != heads * (dn + dv) || dn % 8 ||
      dv % 8 || rot.size(2) % 8 || rot.size(2) > 512 || !aligned(kv) || !aligned(rot))
    return py::none();
  variable_list y;
  {
    py::gil_scoped_release nogil;
    if (at::GradMode::is_enabled() && (recording(kv) || recording(rot))) y = MlaPackFn::apply(kv, rot, heads, dn, dv);
    else y = mla_pack_now(kv, rot, heads, dn, dv);
  }
  return py::make_tuple(y[0], y[1]);
}

// The same written to where the caller keeps keys and values (batches any distance apart); false: nothing was written.
bool mla_pack_into(py::handle kv_, py::handle rot_, int64_t heads, int64_t dn, int64_t dv, py::handle k_, py::handle v_) {
  Tensor kv, rot, k, v;
  if (!unobserved() || !unpack(kv_, kv) || !unpack(rot_, rot) || !unpack(k_, k) || !unpack(v_, v) || !plain_rows(kv) ||
      !plain_rows(rot) || !plain(k) || !plain(v) || rot.dim() != 3 || kv.dim() != 3 || k.dim() != 4 || v.dim() != 4)
    return false;
  const int64_t b = rot.size(0), s = rot.size(1), dr = rot.size(2), dk = dn + dr;
  const auto dense = [&](const Tensor& t, int64_t d) {
    return t.sizes() == at::IntArrayRef({b, s, heads, d}) && t.stride(3) == 1 && t.stride(2) == d && t.stride(1) == heads * d &&
           t.stride(0) % 8 == 0 && (b == 1 || t.stride(0) >= s * heads * d) && aligned(t) && t.device() == kv.device();
  };
  if (kv.size(0) != b || kv.size(1) != s || kv.size(2) != heads * (dn + dv) || dn % 8 || dv % 8 || dr % 8 || dr > 512 ||
      b > 65535 || !aligned(kv) || !aligned(rot) || !dense(k, dk) || !dense(v, dv) ||
      (at::GradMode::is_enabled() && (recording(kv) || recording(rot) || recording(k) || recording(v))))
    return false;
  {
    py::gil_scoped_release nogil;
    check(tpb_mla_pack_rows(cptr(kv), cptr(rot), dr, mptr(k), k.stride(0), mptr(v), v.stride(0), (int)b, s, (int)heads, (int)dn,
                            (int)dr, (int)dv, stream()),
          "mla_pack_into");
    for (const Tensor& t : {k, v})
      if (!t.is_inference()) t.unsafeGetTensorImpl()->bump_version();
  }
  return true;
}

// ------------------------------------------------------------------------------------------- without gradients only
py::object embedding(py::handle ids_, py::handle table_) {
  Tensor ids, table, y;
  if (at::GradMode::is_enabled() || !unobserved() || !unpack(ids_, ids) || !unpack(table_, table) || !plain_rows(ids, at::kLong) ||
      !plain_rows(table) || table.dim() != 2 || table.size(1) % 8 || ids.get_device() != table.get_device() || !small(ids.numel()))
    return py::none();
  {
    py::gil_scoped_release nogil;
    auto sizes = ids.sizes().vec();
    sizes.push_back(table.size(1));
    y = empty_as(table, sizes);
    check(tpb_embedding_fwd(cptr(table), static_cast<const long long*>(cptr(ids)), mptr(y), (int)ids.numel(), (int)table.size(1),
                            table.size(0), 0, stream()),
          "embedding_fwd");
  }
  return py::cast(y);
}

// What mla_decode.supported asks for; the tensors as given to it.
bool absorb_args(py::handle q_, py::handle ckv_, py::handle nw_, py::handle kvc_, py::handle pec_, py::handle w_, int64_t heads,
                 int64_t dn, int64_t dv, Tensor& q, Tensor& ckv, Tensor& nw, Tensor& kvc, Tensor& pec, Tensor& w) {
  if (at::GradMode::is_enabled() || !unobserved() || !unpack(q_, q) || !unpack(ckv_, ckv) || !unpack(nw_, nw) ||
      !unpack(kvc_, kvc) || !unpack(pec_, pec) || !unpack(w_, w))
    return false;
  for (const Tensor* t : {&q, &ckv, &nw, &kvc, &pec, &w})
    if (!plain_rows(*t) || !aligned(*t)) return false;
  if (q.dim() != 3 || ckv.dim() != 3 || kvc.dim() != 3 || pec.dim() != 3) return false;
  const int64_t b = q.size(0), c = kvc.size(2), dr = pec.size(2);
  return q.size(1) == 1 && b <= 65535 && dv <= 4096 && dr == 64 && c % 64 == 0 && c >= 64 && c <= 512 && dn % 8 == 0 && dn >= 8 &&
         dn <= 512 && q.size(2) == heads * (dn + dr) && ckv.size(0) == b && ckv.size(1) == 1 && ckv.size(2) == c + dr &&
         nw.numel() == c && w.size(-1) == c && w.numel() == heads * (dn + dv) * c && kvc.size(0) >= b && pec.size(0) >= b;
}

bool absorb_supported(py::handle q_, py::handle ckv_, py::handle nw_, py::handle kvc_, py::handle pec_, py::handle w_,
                      int64_t heads, int64_t dn, int64_t dr, int64_t dv, int64_t c) {
  Tensor q, ckv, nw, kvc, pec, w;
  return absorb_args(q_, ckv_, nw_, kvc_, pec_, w_, heads, dn, dv, q, ckv, nw, kvc, pec, w) && pec.size(2) == dr && kvc.size(2) == c;
}

// One decode step over the compressed cache; see mla_decode.absorb_step.
py::object absorb_step(py::handle q_, py::handle ckv_, py::handle nw_, double eps, py::handle cos_, py::handle sin_, int64_t pos,
                       py::handle kvc_, py::handle pec_, py::handle w_, int64_t heads, int64_t dn, int64_t dv, double scale,
                       bool interleaved) {
  Tensor q, ckv, nw, cos, sin, kvc, pec, w, out;
  if (!absorb_args(q_, ckv_, nw_, kvc_, pec_, w_, heads, dn, dv, q, ckv, nw, kvc, pec, w) || !unpack(cos_, cos) || !unpack(sin_, sin))
    return py::none();
  const int64_t b = q.size(0), c = kvc.size(2), dr = pec.size(2);
  if (pos < 0 || kvc.size(1) <= pos || pec.size(1) <= pos || !plain_rows(cos, at::kFloat) || !plain_rows(sin, at::kFloat) ||
      cos.dim() != 2 || sin.dim() != 2 || cos.size(0) <= pos || sin.size(0) <= pos || cos.size(1) != 32 || sin.size(1) != 32)
    return py::none();
  {
    py::gil_scoped_release nogil;
    out = empty_as(q, {b, 1, heads * dv});
    const int64_t ranges = tpb_mla_decode_ranges((int)b, (int)heads, (int)pos + 1);
    Tensor scratch = empty_like_type(q, {b * heads * (c + ranges * (c + 2))}, at::kFloat);
    float* base = static_cast<float*>(mptr(scratch));
    float* part_o = base + b * heads * c;
    check(tpb_mla_decode(mptr(q), cptr(ckv), cptr(nw), static_cast<const float*>(cptr(cos)), static_cast<const float*>(cptr(sin)),
                         mptr(kvc), mptr(pec), kvc.stride(0), pec.stride(0), cptr(w), mptr(out), base, part_o,
                         part_o + b * heads * ranges * c, (int)b, (int)heads, (int)dn, (int)dv, (int)c, (int)dr, (int)pos,
                         (float)scale, (float)eps, interleaved, (int)ranges, stream()),
          "mla_decode");
  }
  return py::cast(out);
}

// fp32 logits of bf16 rows; see functional.linear_f32.
py::object linear_f32(py::handle x_, py::handle w_) {
  Tensor x, w, y;
  if (!unobserved() || !unpack(x_, x) || !unpack(w_, w) || !plain(x) || !plain_rows(w) || x.dim() != 2 || w.dim() != 2 ||
      x.numel() == 0 || x.stride(1) != 1 || x.stride(0) % 8 || x.size(1) != w.size(1) || w.size(1) % 8 || w.size(0) % 8 ||
      !aligned(x) || !aligned(w) || !small(x.size(0)) || !small(w.size(0)) ||
      (at::GradMode::is_enabled() && (recording(x) || recording(w))))
    return py::none();
  {
    py::gil_scoped_release nogil;
    const int64_t t = x.size(0), n = w.size(0), k = w.size(1);
    y = empty_like_type(x, {t, n}, at::kFloat);
    check(tpb_linear_f32(cptr(x), cptr(w), static_cast<float*>(mptr(y)), (int)t, (int)n, (int)k, t > 1 ? x.stride(0) : k, k, n,
                         stream()),
          "linear_f32");
  }
  return py::cast(y);
}

// (weights, indices, scores); see moe._router_forward.
py::object router_topk(py::handle lg_, py::handle bias_, int64_t k, int64_t mode, int64_t n_group, int64_t topk_group,
                       bool norm_topk, double scale) {
  Tensor lg, bias, w, idx, scores;
  if (at::GradMode::is_enabled() || !unobserved() || !unpack(lg_, lg) || !unpack(bias_, bias)) return py::none();
  const bool bias16 = bias.defined() && plain_rows(bias);
  if (!(plain_rows(lg, at::kFloat) || plain_rows(lg)) || lg.dim() != 2 || lg.size(1) > 256 || k < 1 || k > lg.size(1) ||
      !small(lg.size(0)) || (bias.defined() && (!(bias16 || plain_rows(bias, at::kFloat)) || bias.numel() != lg.size(1))))
    return py::none();
  {
    py::gil_scoped_release nogil;
    const int64_t t = lg.size(0), e = lg.size(1);
    w = empty_like_type(lg, {t, k}, at::kFloat);
    idx = empty_like_type(lg, {t, k}, at::kInt);
    scores = empty_like_type(lg, {t, e}, at::kFloat);
    check(tpb_router_topk(cptr(lg), (lg.scalar_type() == at::kBFloat16 ? 1 : 0) + (bias16 ? 2 : 0), cptr(bias),
                          static_cast<float*>(mptr(w)), static_cast<int*>(mptr(idx)), static_cast<float*>(mptr(scores)), (int)t,
                          (int)e, (int)k, (int)mode, (int)n_group, (int)topk_group, norm_topk, (float)scale, stream()),
          "router_topk");
  }
  return py::make_tuple(w, idx, scores);
}

// Routed experts with a handful of rows each; see moe.grouped_mlp_few_rows.
py::object grouped_mlp_few_rows(py::handle x_, py::handle rw_, py::handle idx_, py::handle wg_, py::handle wu_, py::handle wd_,
                                bool fused, int64_t align) {
  Tensor x, rw, idx, wg, wu, wd, y;
  if (at::GradMode::is_enabled() || !unobserved() || !unpack(x_, x) || !unpack(rw_, rw) || !unpack(idx_, idx) || !unpack(wg_, wg) ||
      !unpack(wu_, wu) || !unpack(wd_, wd) || !plain_rows(x) || !plain_rows(rw, at::kFloat) || !plain_rows(idx, at::kInt) ||
      !plain_rows(wg) || !plain_rows(wd) || (!fused && !plain_rows(wu)))
    return py::none();
  if (x.dim() != 2 || idx.dim() != 2 || wg.dim() != 3 || wd.dim() != 3 || !aligned(wg) || !aligned(wd) || (!fused && !aligned(wu)))
    return py::none();
  const int64_t t = idx.size(0), k = idx.size(1), e = wg.size(0), d = x.size(1), f = wd.size(1), n = t * k;
  if (x.size(0) != t || rw.numel() != n || wd.size(0) != e || wd.size(2) != d || wg.size(1) != d ||
      wg.size(2) != (fused ? 2 * f : f) || (!fused && wu.sizes() != wg.sizes()) || d % 64 || f % 64 || e > 256)
    return py::none();
  const int64_t hit = std::min(e, n), m = std::max(align, (n + (align - 1) * hit + align - 1) / align * align);
  if (!small(m)) return py::none();
  {
    py::gil_scoped_release nogil;
    Tensor ints = empty_as(idx, {e + (e + 1) + n + m + m / align}), pair = empty_like_type(idx, {m}, at::kLong);
    int *counts = static_cast<int*>(mptr(ints)), *off = counts + e, *dest = off + e + 1, *src = dest + n, *tile = src + m;
    check(tpb_moe_plan(iptr(idx), (int)t, (int)k, (int)e, (int)m, (int)align, counts, off, dest, src,
                       static_cast<long long*>(mptr(pair)), tile, stream()),
          "moe_plan");
    Tensor xg = empty_as(x, {m, d}), act = empty_as(x, {m, f}), rows = empty_as(x, {m, d});
    y = empty_as(x, {t, d});
    check(tpb_moe_gather_real(cptr(x), src, mptr(xg), m, (int)d, stream()), "moe_gather_real");
    check(tpb_grouped_gemm_skinny_bf16(cptr(xg), cptr(wg), fused ? nullptr : cptr(wu), mptr(act), (int)m, (int)(2 * f), (int)d,
                                       (int)e, d, wg.stride(1), wg.stride(0), f, 1, TPB_EPI_SWIGLU, tile, (int)hit, (int)align,
                                       stream()),
          "grouped_gemm_skinny gate/up");
    check(tpb_grouped_gemm_skinny_bf16(cptr(act), cptr(wd), nullptr, mptr(rows), (int)m, (int)d, (int)f, (int)e, f, d,
                                       wd.stride(0), d, 1, TPB_EPI_BF16, tile, (int)hit, (int)align, stream()),
          "grouped_gemm_skinny down");
    check(tpb_moe_combine(cptr(rows), dest, static_cast<const float*>(cptr(rw)), mptr(y), t, (int)k, (int)d, stream()),
          "moe_combine");
  }
  return py::cast(y);
}

}  // namespace

PYBIND11_MODULE(_tpb_torch, m) {
  m.def("configure", [](py::object check_fn, py::object late_wgrads, py::object late_norm) {
    g_check = check_fn.release().ptr();
    g_late_wgrads = late_wgrads.release().ptr();
    g_late_norm = late_norm.release().ptr();
    g_main_grad = PyUnicode_InternFromString("main_grad");
  });
  m.def("launch_count", []() { return g_launches.load(); });
  m.def("linear", &linear);
  m.def("linear_pair", &linear_pair);
  m.def("linear_swiglu", &linear_swiglu);
  m.def("swiglu_mlp", &swiglu_mlp);
  m.def("rms_norm", &rms_norm);
  m.def("rms_norm_residual", &rms_norm_residual);
  m.def("rope", &rope);
  m.def("attention_qkv", &attention_qkv);
  m.def("attention", &attention);
  m.def("latent_split", &latent_split);
  m.def("latent_split_rope", &latent_split_rope);
  m.def("mla_pack", &mla_pack);
  m.def("mla_pack_into", &mla_pack_into);
  m.def("embedding", &embedding);
  m.def("absorb_supported", &absorb_supported);
  m.def("absorb_step", &absorb_step);
  m.def("linear_f32", &linear_f32);
  m.def("router_topk", &router_topk);
  m.def("grouped_mlp_few_rows", &grouped_mlp_few_rows);
}
