// Native form of the operator front-end for the calls a program makes every step: contiguous tensors of one
// type on the current device.  ops.py's Python form costs 25 to 30 us per call (attribute look-ups,
// torch functions and a ctypes call with 17 arguments), several times what the decode kernels take; this
// one 4 to 7 us.  Anything out of the ordinary - a cast, a copy, a broadcast, an error to report - makes a
// function here return None, and the caller goes through the Python form, which handles all of it.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/b200q.h"

namespace {

using at::Tensor;

// ---- scratch buffers: owned and grown by ops._workspaces, known here by address
struct Scratch {
  int dev, op;
  void* stream;
  void* ptr;
  size_t bytes;
};
std::vector<Scratch> g_scratch;   // a handful of (device, stream, operator) triples; guarded by the GIL

const Scratch* find_scratch(int dev, void* stream, int op, size_t need) {
  for (const Scratch& s : g_scratch)
    if (s.dev == dev && s.stream == stream && s.op == op) return s.bytes >= need ? &s : nullptr;
  return nullptr;
}

// B200Q_CHECK_STATUS=1 (read on every call, as the Python form does): status checks live there.
bool checked() {
  const char* e = getenv("B200Q_CHECK_STATUS");
  return e && e[0] == '1' && e[1] == 0;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return B200Q_F32;
    case at::kHalf: return B200Q_F16;
    case at::kBFloat16: return B200Q_BF16;
    default: return -1;
  }
}

// A plain torch.Tensor (or Parameter) argument; nullptr for anything else.
const Tensor* tensor(PyObject* o) {
  return THPVariable_CheckTypeExact(Py_TYPE(o)) ? &THPVariable_Unpack(o) : nullptr;
}
bool integer(PyObject* o, int dflt, int* out) {
  if (o == Py_None) { *out = dflt; return true; }
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow != 0 || v < INT_MIN || v > INT_MAX) return false;   // the Python form says what is wrong with it
  *out = (int)v;
  return true;
}
bool affine(PyObject* o) { return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, "affine") == 0; }

// Quantized matrix operands that need no cast and no copy: w uint32, scales and biases of type `t` and of one
// shape, all contiguous on `dev`.
bool plain_weights(const Tensor& w, const Tensor& s, const Tensor& b, at::ScalarType t, at::Device dev, int group, int bits) {
  if (w.scalar_type() != at::kUInt32 || s.scalar_type() != t || b.scalar_type() != t) return false;
  if (w.device() != dev || s.device() != dev || b.device() != dev) return false;
  const int64_t nd = w.dim();
  if (nd < 2 || s.dim() != nd || b.dim() != nd) return false;
  for (int64_t i = 0; i < nd - 1; ++i)
    if (s.size(i) != w.size(i) || b.size(i) != w.size(i)) return false;
  if (s.size(nd - 1) != b.size(nd - 1) || w.size(nd - 1) * 32 % bits != 0 || w.size(nd - 1) * 32 / bits != s.size(nd - 1) * group) return false;
  return w.is_contiguous() && s.is_contiguous() && b.is_contiguous();
}
bool current(at::Device dev) { return dev.is_cuda() && dev.index() == c10::cuda::current_device(); }
bool params_ok(int group, int bits) { return (group == 32 || group == 64 || group == 128) && bits >= 2 && bits <= 8 && bits != 7; }

PyObject* none() { Py_RETURN_NONE; }

// ---- quantized_matmul.  False: not an ordinary call (or the library refused it): take the Python form.
bool qmm_run(const Tensor& x, const Tensor& w, const Tensor& s, const Tensor& b, bool transpose, int group, int bits, Tensor* y) {
  const at::ScalarType t = x.scalar_type();
  const int dt = dtype_code(t);
  const at::Device dev = x.device();
  if (dt < 0 || !params_ok(group, bits) || !current(dev) || x.dim() < 2 || w.dim() != 2 || !x.is_contiguous() ||
      !plain_weights(w, s, b, t, dev, group, bits) || checked())
    return false;
  const int64_t inner = w.size(1) * 32 / bits;
  const int64_t K = x.size(-1), M = K ? x.numel() / K : 0, N = transpose ? w.size(0) : inner;
  if (M == 0 || N == 0 || K != (transpose ? inner : w.size(0))) return false;
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const size_t need = b200q_qmm_workspace_bytes(dt, 1, M, N, K, group, bits, transpose);
  const Scratch* ws = find_scratch(dev.index(), stream, 0, need);
  if (!ws) return false;
  c10::SmallVector<int64_t, 6> size(x.sizes().begin(), x.sizes().end());
  size.back() = N;
  *y = at::detail::empty_cuda(size, t, dev, std::nullopt);
  return b200q_qmm(x.data_ptr(), static_cast<const uint32_t*>(w.data_ptr()), s.data_ptr(), b.data_ptr(), y->data_ptr(), dt, 1,
                   M, N, K, group, bits, transpose, 0, ws->ptr, ws->bytes, stream) == B200Q_OK;
}

// (x, w, scales, biases, transpose, group_size, bits, mode)
bool qmm_args(PyObject* const* a, Py_ssize_t n, const Tensor* (&t)[4], bool* transpose, int* group, int* bits) {
  if (n != 8) return false;
  for (int i = 0; i < 4; ++i)
    if (!(t[i] = tensor(a[i]))) return false;
  if (!PyBool_Check(a[4]) || !integer(a[5], 64, group) || !integer(a[6], 4, bits) || !affine(a[7])) return false;
  *transpose = a[4] == Py_True;
  return true;
}

PyObject* py_qmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor* t[4];
  bool transpose;
  int group, bits;
  Tensor y;
  if (!qmm_args(a, n, t, &transpose, &group, &bits)) return none();
  if (!qmm_run(*t[0], *t[1], *t[2], *t[3], transpose, group, bits, &y)) return none();
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// ---- quantize, dequantize
PyObject* py_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {   // (w, group_size, bits, mode)
  HANDLE_TH_ERRORS
  int group, bits;
  const Tensor* w;
  if (n != 4 || !(w = tensor(a[0])) || !integer(a[1], 64, &group) || !integer(a[2], 4, &bits) || !affine(a[3])) return none();
  const at::ScalarType t = w->scalar_type();
  const int dt = dtype_code(t);
  const at::Device dev = w->device();
  if (dt < 0 || !params_ok(group, bits) || !current(dev) || w->dim() < 2 || !w->is_contiguous() || w->numel() == 0) return none();
  const int64_t K = w->size(-1);
  if (K % group != 0) return none();
  c10::SmallVector<int64_t, 6> size(w->sizes().begin(), w->sizes().end());
  size.back() = K * bits / 32;
  Tensor wq = at::detail::empty_cuda(size, at::kUInt32, dev, std::nullopt);
  size.back() = K / group;
  Tensor s = at::detail::empty_cuda(size, t, dev, std::nullopt), b = at::detail::empty_cuda(size, t, dev, std::nullopt);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  if (b200q_quantize(w->data_ptr(), dt, w->numel() / K, K, group, bits, static_cast<uint32_t*>(wq.data_ptr()), s.data_ptr(),
                     b.data_ptr(), stream) != B200Q_OK)
    return none();
  PyObject* out = PyTuple_New(3);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(wq)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(s)));
  PyTuple_SET_ITEM(out, 2, THPVariable_Wrap(std::move(b)));
  return out;
  END_HANDLE_TH_ERRORS
}

PyObject* py_dequantize(PyObject*, PyObject* const* a, Py_ssize_t n) {   // (w, scales, biases, group_size, bits, mode)
  HANDLE_TH_ERRORS
  int group, bits;
  const Tensor *w, *s, *b;
  if (n != 6 || !(w = tensor(a[0])) || !(s = tensor(a[1])) || !(b = tensor(a[2])) || !integer(a[3], 64, &group) ||
      !integer(a[4], 4, &bits) || !affine(a[5]))
    return none();
  const at::ScalarType t = s->scalar_type();
  const int dt = dtype_code(t);
  const at::Device dev = w->device();
  if (dt < 0 || !params_ok(group, bits) || !current(dev) || !plain_weights(*w, *s, *b, t, dev, group, bits) || w->numel() == 0)
    return none();
  const int64_t words = w->size(-1), K = words * 32 / bits;
  c10::SmallVector<int64_t, 6> size(w->sizes().begin(), w->sizes().end());
  size.back() = K;
  Tensor out = at::detail::empty_cuda(size, t, dev, std::nullopt);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  if (b200q_dequantize(static_cast<const uint32_t*>(w->data_ptr()), s->data_ptr(), b->data_ptr(), dt, w->numel() / words, K, group,
                       bits, out.data_ptr(), stream) != B200Q_OK)
    return none();
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// ---- quantized_matmul with a gradient for x alone (frozen scales and biases)
struct QmmFn : public torch::autograd::Function<QmmFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& s, const Tensor& b,
                        bool transpose, int64_t group, int64_t bits, Tensor* y) {
    ctx->save_for_backward({w, s, b});
    ctx->saved_data["transpose"] = transpose;
    ctx->saved_data["group"] = group;
    ctx->saved_data["bits"] = bits;
    return *y;   // by address: a result passed as a tensor would come back as a view of itself
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const bool transpose = ctx->saved_data["transpose"].toBool();
    const int64_t group = ctx->saved_data["group"].toInt(), bits = ctx->saved_data["bits"].toInt();
    const Tensor dy = grads[0].contiguous();
    Tensor dx;
    pybind11::gil_scoped_acquire gil;   // the scratch table, and the Python form
    if (!qmm_run(dy, saved[0], saved[1], saved[2], !transpose, (int)group, (int)bits, &dx)) {
      const auto ops = pybind11::module_::import("mlx_b200.ops");
      auto wrap = [](const Tensor& t) { return pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t)); };
      pybind11::object r = ops.attr("quantized_matmul")(wrap(dy), wrap(saved[0]), wrap(saved[1]), wrap(saved[2]), !transpose, group, bits);
      dx = THPVariable_Unpack(r.ptr());
    }
    return {dx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

PyObject* py_qmm_grad(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor* t[4];
  bool transpose;
  int group, bits;
  Tensor y;
  if (!qmm_args(a, n, t, &transpose, &group, &bits)) return none();
  if (t[2]->requires_grad() || t[3]->requires_grad()) return none();
  for (const Tensor* u : t)   // forward-mode differentiation: the Python form's autograd.Function says that it has none
    if (u->_fw_grad(0).defined()) return none();
  {
    at::AutoDispatchBelowAutograd below;
    if (!qmm_run(*t[0], *t[1], *t[2], *t[3], transpose, group, bits, &y)) return none();
  }
  if (t[0]->requires_grad() && at::GradMode::is_enabled())
    y = QmmFn::apply(*t[0], *t[1], *t[2], *t[3], transpose, (int64_t)group, (int64_t)bits, &y);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// ---- gather_qmm and the gated expert layer
// An index operand as a view over the pairs: right-aligned to four dimensions.  `t` null: the default index, which is
// the offset into `lead` (the batch dimensions of the operand it selects from).
struct View {
  b200q_index v;
  int64_t shape[4];
};
bool make_view(const Tensor* t, at::IntArrayRef lead, at::Device dev, View* out) {
  for (int d = 0; d < 4; ++d) { out->shape[d] = 1; out->v.stride[d] = 0; }
  out->v.data = nullptr;
  out->v.elem_bytes = 4;
  const int64_t nd = t ? t->dim() : (int64_t)lead.size();
  if (nd > 4) return false;
  if (t) {
    const at::ScalarType k = t->scalar_type();
    if (t->device() != dev || (k != at::kLong && k != at::kInt && k != at::kUInt32)) return false;
    if (t->numel() == 0) return false;
    out->v.data = t->data_ptr();
    out->v.elem_bytes = k == at::kLong ? 8 : 4;
    for (int64_t d = 0; d < nd; ++d) {
      out->shape[4 - nd + d] = t->size(d);
      out->v.stride[4 - nd + d] = t->size(d) == 1 ? 0 : t->stride(d);
    }
  } else {
    int64_t st = 1;
    for (int64_t d = nd - 1; d >= 0; --d) {
      out->shape[4 - nd + d] = lead[d];
      out->v.stride[4 - nd + d] = lead[d] == 1 ? 0 : st;
      st *= lead[d];
    }
  }
  return true;
}
// The pairs' shape (and the output's leading dimensions); false where the views do not broadcast.
bool broadcast(View* a, View* b, int64_t nd_a, int64_t nd_b, int64_t shape[4], int64_t* n, c10::SmallVector<int64_t, 6>* lead) {
  *n = 1;
  for (int d = 0; d < 4; ++d) {
    if (a->shape[d] != b->shape[d] && a->shape[d] != 1 && b->shape[d] != 1) return false;
    shape[d] = a->shape[d] == 1 ? b->shape[d] : a->shape[d];
    *n *= shape[d];
  }
  lead->clear();
  for (int d = 4 - (int)std::max(nd_a, nd_b); d < 4; ++d) lead->push_back(shape[d]);
  return true;
}
int64_t product(at::IntArrayRef v) {
  int64_t n = 1;
  for (int64_t x : v) n *= x;
  return n;
}
// Index argument: None, or a plain tensor.
bool index_arg(PyObject* o, const Tensor** t) {
  if (o == Py_None) { *t = nullptr; return true; }
  return (*t = tensor(o)) != nullptr;
}

// (x, w, scales, biases, lhs_indices, rhs_indices, transpose, group_size, bits, mode)
PyObject* py_gather(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *w, *s, *b, *li, *ri;
  int group, bits;
  if (n != 10 || !(x = tensor(a[0])) || !(w = tensor(a[1])) || !(s = tensor(a[2])) || !(b = tensor(a[3])) || !index_arg(a[4], &li) ||
      !index_arg(a[5], &ri) || (!li && !ri) || a[6] != Py_True || !integer(a[7], 64, &group) || !integer(a[8], 4, &bits) ||
      !affine(a[9]))
    return none();
  const at::Device dev = x->device();
  if (x->scalar_type() != at::kBFloat16 || !params_ok(group, bits) || !current(dev) || x->dim() < 2 || w->dim() < 3 ||
      !x->is_contiguous() || !plain_weights(*w, *s, *b, at::kBFloat16, dev, group, bits) || checked())
    return none();
  const int64_t M = x->size(-2), K = x->size(-1), N = w->size(-2), x_batch = product(x->sizes().slice(0, x->dim() - 2)),
                E = product(w->sizes().slice(0, w->dim() - 2));
  if (w->size(-1) * 32 / bits != K || M == 0 || N == 0 || K == 0 || x_batch == 0 || E == 0) return none();
  View l, r;
  int64_t shape[4], n_idx;
  c10::SmallVector<int64_t, 6> size;
  const auto xl = x->sizes().slice(0, x->dim() - 2), wl = w->sizes().slice(0, w->dim() - 2);
  if (!make_view(li, xl, dev, &l) || !make_view(ri, wl, dev, &r) ||
      !broadcast(&l, &r, li ? li->dim() : (int64_t)xl.size(), ri ? ri->dim() : (int64_t)wl.size(), shape, &n_idx, &size))
    return none();
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const Scratch* ws = find_scratch(dev.index(), stream, 1, b200q_gather_qmm_workspace_bytes(B200Q_BF16, n_idx, x_batch, E, M, N, K, group, bits, 1));
  if (!ws) return none();
  size.push_back(M);
  size.push_back(N);
  Tensor y = at::detail::empty_cuda(size, at::kBFloat16, dev, std::nullopt);
  if (b200q_gather_qmm_indexed(x->data_ptr(), static_cast<const uint32_t*>(w->data_ptr()), s->data_ptr(), b->data_ptr(), &l.v, &r.v,
                               shape, y.data_ptr(), B200Q_BF16, x_batch, E, M, N, K, group, bits, ws->ptr, ws->bytes, stream) != B200Q_OK)
    return none();
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// A (w, scales, biases) triple of plain tensors.
bool triple(PyObject* o, const Tensor* (&t)[3]) {
  if (!(PyTuple_CheckExact(o) || PyList_CheckExact(o)) || PySequence_Fast_GET_SIZE(o) != 3) return false;
  for (int i = 0; i < 3; ++i)
    if (!(t[i] = tensor(PySequence_Fast_GET_ITEM(o, i)))) return false;
  return true;
}

// (x, gate, up, down, rhs_indices, lhs_indices, group_size, bits)
PyObject* py_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const Tensor *x, *g[3], *u[3], *d[3], *li, *ri;
  int group, bits;
  if (n != 8 || !(x = tensor(a[0])) || !triple(a[1], g) || !triple(a[2], u) || !triple(a[3], d) || !index_arg(a[4], &ri) || !ri ||
      !index_arg(a[5], &li) || !integer(a[6], 64, &group) || !integer(a[7], 4, &bits))
    return none();
  const at::Device dev = x->device();
  if (x->scalar_type() != at::kBFloat16 || !params_ok(group, bits) || !current(dev) || x->dim() < 2 || g[0]->dim() < 3 ||
      !x->is_contiguous() || checked())
    return none();
  for (const auto& t : {g, u, d})
    if (!plain_weights(*t[0], *t[1], *t[2], at::kBFloat16, dev, group, bits)) return none();
  const int64_t M = x->size(-2), K1 = x->size(-1), H = g[0]->size(-2), N2 = d[0]->size(-2),
                x_batch = product(x->sizes().slice(0, x->dim() - 2)), E = product(g[0]->sizes().slice(0, g[0]->dim() - 2));
  if (g[0]->sizes() != u[0]->sizes() || g[0]->size(-1) * 32 / bits != K1 || d[0]->size(-1) * 32 / bits != H ||
      g[0]->dim() != d[0]->dim() || g[0]->sizes().slice(0, g[0]->dim() - 2) != d[0]->sizes().slice(0, d[0]->dim() - 2) || M == 0 ||
      K1 == 0 || H == 0 || N2 == 0 || x_batch == 0 || E == 0)
    return none();
  View l, r;
  int64_t shape[4], n_idx;
  c10::SmallVector<int64_t, 6> size;
  const auto xl = x->sizes().slice(0, x->dim() - 2);
  if (!make_view(li, xl, dev, &l) || !make_view(ri, xl, dev, &r) ||
      !broadcast(&l, &r, li ? li->dim() : (int64_t)xl.size(), ri->dim(), shape, &n_idx, &size))
    return none();
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const Scratch* ws = find_scratch(dev.index(), stream, 1, b200q_gather_qmm_swiglu_workspace_bytes(n_idx, E, M, H, K1));
  if (!ws) return none();
  size.push_back(M);
  size.push_back(N2);
  Tensor y = at::detail::empty_cuda(size, at::kBFloat16, dev, std::nullopt);
  auto w = [](const Tensor* t) { return static_cast<const uint32_t*>(t->data_ptr()); };
  if (b200q_gather_qmm_swiglu_indexed(x->data_ptr(), w(g[0]), g[1]->data_ptr(), g[2]->data_ptr(), w(u[0]), u[1]->data_ptr(),
                                      u[2]->data_ptr(), w(d[0]), d[1]->data_ptr(), d[2]->data_ptr(), &l.v, &r.v, shape, y.data_ptr(),
                                      B200Q_BF16, x_batch, E, M, H, K1, N2, group, bits, ws->ptr, ws->bytes, stream) != B200Q_OK)
    return none();
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// (device index, stream, operator, address, bytes): ops._workspaces has a new buffer
PyObject* py_scratch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) { PyErr_SetString(PyExc_TypeError, "scratch takes five arguments"); return nullptr; }
  const Scratch s{(int)PyLong_AsLong(a[0]), (int)PyLong_AsLong(a[2]), PyLong_AsVoidPtr(a[1]), PyLong_AsVoidPtr(a[3]), PyLong_AsSize_t(a[4])};
  if (PyErr_Occurred()) return nullptr;
  for (Scratch& g : g_scratch)
    if (g.dev == s.dev && g.stream == s.stream && g.op == s.op) { g = s; Py_RETURN_NONE; }
  g_scratch.push_back(s);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"qmm", (PyCFunction)(void (*)(void))py_qmm, METH_FASTCALL, nullptr},
    {"qmm_grad", (PyCFunction)(void (*)(void))py_qmm_grad, METH_FASTCALL, nullptr},
    {"quantize", (PyCFunction)(void (*)(void))py_quantize, METH_FASTCALL, nullptr},
    {"dequantize", (PyCFunction)(void (*)(void))py_dequantize, METH_FASTCALL, nullptr},
    {"gather", (PyCFunction)(void (*)(void))py_gather, METH_FASTCALL, nullptr},
    {"swiglu", (PyCFunction)(void (*)(void))py_swiglu, METH_FASTCALL, nullptr},
    {"scratch", (PyCFunction)(void (*)(void))py_scratch, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_front", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front() { return PyModule_Create(&module); }
