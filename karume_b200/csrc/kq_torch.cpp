// The Python calls of the serving loop as one native step each: argument checks, the output
// allocation and the C-ABI call (include/kq.h), for torch tensors.
//
// A small linear is bound by the host: 9.0 us per call through Python checks (1.0), torch.empty
// (2.4, and 1 for its release), ctypes conversions (0.7) and the launch (2.7), where the kernel
// takes 4.  Here everything but the launch is about 1 us.
//
// Every function returns the result, an int (the kq_status of a call the library refused), or None
// when an argument is not of the plain form it handles (then the Python method goes on with its
// own checks and conversions, and raises what they raise).  A C++ exception inside one (an output that
// cannot be allocated, a tensor without memory) leaves as the Python exception torch makes of it.
#define PY_SSIZE_T_CLEAN
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <Python.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <exception>

namespace {

// Addresses of the library's entry points, handed over once (bind): this module does not link libkq,
// it calls the one the ctypes layer has loaded.
using LinearFn = int (*)(void*, uint64_t, uint64_t, int, uint64_t, uint64_t, uint32_t);
using FusedFn = int (*)(void*, uint32_t, const uint64_t*, uint64_t, int, uint64_t, float, const uint64_t*, uint64_t, const uint64_t*, uint32_t,
                        uint32_t);
using QuantizeFn = int (*)(void*, uint64_t, uint32_t, uint32_t, uint64_t, uint64_t);
using A8Fn = int (*)(void*, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint32_t);
using EmbeddingFn = int (*)(void*, uint64_t, uint64_t, uint32_t, uint64_t);
LinearFn g_linear = nullptr;
FusedFn g_fused = nullptr;
QuantizeFn g_quantize = nullptr;
A8Fn g_a8 = nullptr;
EmbeddingFn g_embedding = nullptr;

constexpr int kMaxMulti = 4;

// 0 / 1 / 2 = KQ_F32 / KQ_F16 / KQ_BF16, -1: not an activation type
int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kHalf: return 1;
    case at::kBFloat16: return 2;
    default: return -1;
  }
}
bool plain(const at::Tensor& t) { return t.is_cuda() && t.is_contiguous(); }
uint64_t ptr(const at::Tensor& t) { return reinterpret_cast<uint64_t>(t.data_ptr()); }
bool tensor_of(PyObject* o, const at::Tensor** out) {
  if (!THPVariable_Check(o)) return false;
  *out = &THPVariable_Unpack(o);
  return true;
}
at::Tensor empty_like_lead(const at::Tensor& x, int64_t last, at::ScalarType type) {
  c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = last;
  return at::detail::empty_cuda(shape, type, x.device(), c10::nullopt);
}
PyObject* status_of(int rc) { return PyLong_FromLong(rc); }
#define KQ_NONE Py_RETURN_NONE

// The library call while other Python threads run; the lock is back before anything, an exception too, goes on.
template <typename Call>
int without_gil(Call call) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  return call();
}

PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "bind takes five addresses");
    return nullptr;
  }
  g_linear = reinterpret_cast<LinearFn>(PyLong_AsVoidPtr(a[0]));
  g_fused = reinterpret_cast<FusedFn>(PyLong_AsVoidPtr(a[1]));
  g_quantize = reinterpret_cast<QuantizeFn>(PyLong_AsVoidPtr(a[2]));
  g_a8 = reinterpret_cast<A8Fn>(PyLong_AsVoidPtr(a[3]));
  g_embedding = reinterpret_cast<EmbeddingFn>(PyLong_AsVoidPtr(a[4]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// linear(ctx, handle, n, k, x, bias, out)
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 7 || a[0] == Py_None) KQ_NONE;
  const int64_t n = PyLong_AsLongLong(a[2]), k = PyLong_AsLongLong(a[3]);
  const at::Tensor *x, *bias, *given = nullptr;
  if (!tensor_of(a[4], &x) || !tensor_of(a[5], &bias) || (a[6] != Py_None && !tensor_of(a[6], &given))) KQ_NONE;
  const int type = dtype_code(*x);
  if (type < 0 || !plain(*x) || x->dim() < 1 || x->size(-1) != k || k == 0 || bias->scalar_type() != at::kFloat || bias->dim() != 1 ||
      bias->size(0) != n)
    KQ_NONE;
  at::Tensor made;
  if (given == nullptr) made = empty_like_lead(*x, n, at::kFloat);
  const at::Tensor& out = given != nullptr ? *given : made;
  void* ctx = PyLong_AsVoidPtr(a[0]);
  const uint64_t handle = PyLong_AsUnsignedLongLong(a[1]);
  const uint64_t px = ptr(*x), pb = ptr(*bias), po = ptr(out);
  const uint32_t m = static_cast<uint32_t>(x->numel() / k);
  const int rc = without_gil([&] { return g_linear(ctx, handle, px, type, pb, po, m); });
  if (rc != 0) return status_of(rc);
  if (given != nullptr) return Py_NewRef(a[6]);
  return THPVariable_Wrap(std::move(made));
}

// linear_fused(ctx, handles, k, x, biases, outs, norm_weight, eps, residual, flags): `outs` a list of tensors
PyObject* linear_fused(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 10 || a[0] == Py_None) KQ_NONE;
  PyObject *handles = a[1], *biases = a[4], *outs = a[5];
  if (!PyList_CheckExact(handles) || !PyList_CheckExact(biases) || !PyList_CheckExact(outs)) KQ_NONE;
  const Py_ssize_t count = PyList_GET_SIZE(handles);
  if (count < 1 || count > kMaxMulti || PyList_GET_SIZE(biases) != count || PyList_GET_SIZE(outs) < 1) KQ_NONE;
  const int64_t k = PyLong_AsLongLong(a[2]);
  const at::Tensor *x, *t, *norm = nullptr, *residual = nullptr;
  if (!tensor_of(a[3], &x) || (a[6] != Py_None && !tensor_of(a[6], &norm)) || (a[8] != Py_None && !tensor_of(a[8], &residual))) KQ_NONE;
  const int type = dtype_code(*x);
  if (type < 0 || !plain(*x) || x->dim() < 1 || x->size(-1) != k || k == 0) KQ_NONE;
  uint64_t w[kMaxMulti] = {}, b[kMaxMulti] = {}, o[kMaxMulti] = {};
  for (Py_ssize_t i = 0; i < count; ++i) {
    w[i] = PyLong_AsUnsignedLongLong(PyList_GET_ITEM(handles, i));
    if (!tensor_of(PyList_GET_ITEM(biases, i), &t)) KQ_NONE;
    b[i] = ptr(*t);
    if (i < PyList_GET_SIZE(outs)) {
      if (!tensor_of(PyList_GET_ITEM(outs, i), &t)) KQ_NONE;
      o[i] = ptr(*t);
    }
  }
  void* ctx = PyLong_AsVoidPtr(a[0]);
  const float eps = static_cast<float>(PyFloat_AsDouble(a[7]));
  const uint32_t flags = static_cast<uint32_t>(PyLong_AsUnsignedLong(a[9]));
  if (PyErr_Occurred()) return nullptr;
  const uint64_t px = ptr(*x), pn = norm != nullptr ? ptr(*norm) : 0, pr = residual != nullptr ? ptr(*residual) : 0;
  const uint32_t m = static_cast<uint32_t>(x->numel() / k);
  const int rc = without_gil([&] { return g_fused(ctx, static_cast<uint32_t>(count), w, px, type, pn, eps, b, pr, o, m, flags); });
  if (rc != 0) return status_of(rc);
  return Py_NewRef(outs);
}

// quantize_rows(ctx, x) -> (q, scale)
PyObject* quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  const at::Tensor* x;
  if (nargs != 2 || a[0] == Py_None || !tensor_of(a[1], &x) || x->scalar_type() != at::kFloat || !plain(*x) || x->dim() < 1) KQ_NONE;
  const int64_t dim = x->size(-1);
  if (dim == 0) KQ_NONE;
  at::Tensor q = at::detail::empty_cuda(x->sizes(), at::kChar, x->device(), c10::nullopt);
  at::Tensor scale = at::detail::empty_cuda(x->sizes().slice(0, x->dim() - 1), at::kFloat, x->device(), c10::nullopt);
  void* ctx = PyLong_AsVoidPtr(a[0]);
  const uint64_t px = ptr(*x), pq = ptr(q), ps = ptr(scale);
  const uint32_t rows = static_cast<uint32_t>(x->numel() / dim);
  const int rc = without_gil([&] { return g_quantize(ctx, px, rows, static_cast<uint32_t>(dim), pq, ps); });
  if (rc != 0) return status_of(rc);
  PyObject *pyq = THPVariable_Wrap(std::move(q)), *pys = THPVariable_Wrap(std::move(scale));
  PyObject* r = pyq != nullptr && pys != nullptr ? PyTuple_Pack(2, pyq, pys) : nullptr;
  Py_XDECREF(pyq);
  Py_XDECREF(pys);
  return r;
}

// linear_a8(ctx, handle, n, k, xq, xs, bias, out)
PyObject* linear_a8(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 8 || a[0] == Py_None) KQ_NONE;
  const int64_t n = PyLong_AsLongLong(a[2]), k = PyLong_AsLongLong(a[3]);
  const at::Tensor *xq, *xs, *bias, *given = nullptr;
  if (!tensor_of(a[4], &xq) || !tensor_of(a[5], &xs) || !tensor_of(a[6], &bias) || (a[7] != Py_None && !tensor_of(a[7], &given))) KQ_NONE;
  if (xq->scalar_type() != at::kChar || !plain(*xq) || xq->dim() < 1 || xq->size(-1) != k || k == 0 || xs->scalar_type() != at::kFloat ||
      xs->numel() != xq->numel() / k || bias->scalar_type() != at::kFloat || bias->numel() != n)
    KQ_NONE;
  at::Tensor made;
  if (given == nullptr) made = empty_like_lead(*xq, n, at::kFloat);
  const at::Tensor& out = given != nullptr ? *given : made;
  void* ctx = PyLong_AsVoidPtr(a[0]);
  const uint64_t handle = PyLong_AsUnsignedLongLong(a[1]);
  const uint64_t pq = ptr(*xq), ps = ptr(*xs), pb = ptr(*bias), po = ptr(out);
  const uint32_t m = static_cast<uint32_t>(xq->numel() / k);
  const int rc = without_gil([&] { return g_a8(ctx, handle, pq, ps, pb, po, m); });
  if (rc != 0) return status_of(rc);
  if (given != nullptr) return Py_NewRef(a[7]);
  return THPVariable_Wrap(std::move(made));
}

// embedding(ctx, handle, k, index, out)
PyObject* embedding(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 5 || a[0] == Py_None) KQ_NONE;
  const int64_t k = PyLong_AsLongLong(a[2]);
  const at::Tensor *index, *given = nullptr;
  if (!tensor_of(a[3], &index) || (a[4] != Py_None && !tensor_of(a[4], &given)) || index->scalar_type() != at::kInt || !plain(*index)) KQ_NONE;
  at::Tensor made;
  if (given == nullptr) {
    c10::SmallVector<int64_t, 8> shape(index->sizes().begin(), index->sizes().end());
    shape.push_back(k);
    made = at::detail::empty_cuda(shape, at::kFloat, index->device(), c10::nullopt);
  }
  const at::Tensor& out = given != nullptr ? *given : made;
  void* ctx = PyLong_AsVoidPtr(a[0]);
  const uint64_t handle = PyLong_AsUnsignedLongLong(a[1]);
  const uint64_t pi = ptr(*index), po = ptr(out);
  const uint32_t rows = static_cast<uint32_t>(index->numel());
  const int rc = without_gil([&] { return g_embedding(ctx, handle, pi, rows, po); });
  if (rc != 0) return status_of(rc);
  if (given != nullptr) return Py_NewRef(a[4]);
  return THPVariable_Wrap(std::move(made));
}

// CPython's frames have no handlers: what is thrown in a call must not leave it.
template <PyObject* (*kCall)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t nargs) {
  try {
    return kCall(self, a, nargs);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

#define KQ_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {KQ_METHOD(bind),      KQ_METHOD(linear),    KQ_METHOD(linear_fused), KQ_METHOD(quantize_rows),
                         KQ_METHOD(linear_a8), KQ_METHOD(embedding), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_kqtorch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__kqtorch() { return PyModule_Create(&module); }
