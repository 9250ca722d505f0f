// Python binding of the calls a decode loop issues step by step.
//
// A projection of one token keeps the GPU busy for about two microseconds.  Checking the
// tensors of such a call in Python, naming the device and the stream through torch's Python
// API and converting the arguments with ctypes takes eight, so a step that issues its
// projections one by one is bound by the host.  The functions here look at the tensors
// directly and call the C ABI.
//
// They take a call only when everything about it is as it should be, and return -1
// otherwise, before anything is launched: the caller then goes through the Python checks,
// which raise what they always raised.  A tensor subclass, a functorch wrapper, a lazy
// conjugate or negation, another device than the current one or a strided view all count as
// "otherwise".  The result is else the status of the C entry point.
//
// The library is not linked: `bind` receives the entry points' addresses, so that the
// binding calls whichever library the Python side has loaded.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/core/DispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../include/cudalm_b200.h"

namespace {

decltype(&cudalm_b200_int4_gemv_bf16) g_gemv = nullptr;
decltype(&cudalm_b200_batch_int4_gemv_bf16) g_batch = nullptr;
decltype(&cudalm_b200_linear_multi) g_multi = nullptr;
decltype(&cudalm_b200_gate_up_silu_bf16) g_gate_up_silu = nullptr;
decltype(&cudalm_b200_linear_residual_bf16) g_residual = nullptr;

PyObject *s_weight, *s_scale, *s_N, *s_K;  // interned attribute names

constexpr int64_t kIntMax = 0x7fffffff;

PyObject* status(int rc) { return PyLong_FromLong(rc); }
PyObject* not_taken() {
  PyErr_Clear();
  return PyLong_FromLong(-1);
}

// The tensor behind `o` when it is an ordinary contiguous CUDA tensor of this type on
// device `dev`; null otherwise.
const at::Tensor* plain(PyObject* o, at::ScalarType type, int dev) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched,
                                            c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                            c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  if (!t.defined() || t.scalar_type() != type || !t.is_cuda() || t.device().index() != dev ||
      t.layout() != at::kStrided || t.key_set().has_any(wrapped) || !t.is_contiguous())
    return nullptr;
  return &t;
}

struct Lin {
  const at::Tensor *weight = nullptr, *scale = nullptr;
  int64_t N = 0, K = 0;
};

bool int_attr(PyObject* o, PyObject* name, int64_t* out) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (!v) return false;
  const bool ok = PyLong_CheckExact(v);
  *out = ok ? PyLong_AsLongLong(v) : -1;
  Py_DECREF(v);
  return ok && *out > 0 && *out <= kIntMax;
}

// weight, scale, N and K of a W4A16Linear, which keeps the tensors alive.
bool read_linear(PyObject* o, int dev, Lin* lin) {
  PyObject* w = PyObject_GetAttr(o, s_weight);
  PyObject* s = w ? PyObject_GetAttr(o, s_scale) : nullptr;
  if (w && s) {
    lin->weight = plain(w, at::kByte, dev);
    lin->scale = plain(s, at::kHalf, dev);
  }
  // borrowed from here on, which needs the object to hold them
  const bool held = w && s && Py_REFCNT(w) > 1 && Py_REFCNT(s) > 1;
  Py_XDECREF(w);
  Py_XDECREF(s);
  if (!held || !lin->weight || !lin->scale) return false;
  if (!int_attr(o, s_N, &lin->N) || !int_attr(o, s_K, &lin->K)) return false;
  return lin->K % 128 == 0 && lin->weight->numel() >= lin->N * (lin->K / 2) &&
         lin->scale->numel() >= lin->N * (lin->K / 128);
}

int64_t rows_of(const at::Tensor& x) { return x.dim() == 1 ? 1 : (x.dim() == 0 ? 0 : x.size(0)); }

const uint8_t* bytes(const at::Tensor* t) { return static_cast<const uint8_t*>(t->data_ptr()); }
uint16_t* halves(const at::Tensor* t) { return static_cast<uint16_t*>(t->data_ptr()); }

void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(); }

// gemv(weight, scales, x, y) and batch(weight, scales, x, y)
PyObject* projection(PyObject* const* a, Py_ssize_t n, bool batched) {
  if (n != 4 || !g_batch) return not_taken();
  try {
    const int dev = c10::cuda::current_device();
    const at::Tensor* w = plain(a[0], at::kByte, dev);
    const at::Tensor* s = plain(a[1], at::kHalf, dev);
    const at::Tensor* x = plain(a[2], at::kBFloat16, dev);
    const at::Tensor* y = plain(a[3], at::kBFloat16, dev);
    if (!w || !s || !x || !y || w->dim() < 2 || (batched && x->dim() < 1)) return not_taken();
    const int64_t N = w->size(0), K = 2 * w->size(1), B = batched ? x->size(0) : 1;
    if (N < 1 || K < 1 || K % 128 || B < 1 || N > kIntMax || K > kIntMax || B > kIntMax) return not_taken();
    if (w->numel() < N * (K / 2) || s->numel() < N * (K / 128) || x->numel() != B * K || y->numel() < B * N)
      return not_taken();
    const uint8_t* wp = bytes(w);
    uint16_t *sp = halves(s), *xp = halves(x), *yp = halves(y);
    void* st = stream_of(dev);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = batched ? g_batch(wp, sp, xp, yp, static_cast<int>(N), static_cast<int>(K), static_cast<int>(B), st)
                 : g_gemv(wp, sp, xp, yp, static_cast<int>(N), static_cast<int>(K), st);
    Py_END_ALLOW_THREADS
    return status(rc);
  } catch (...) {
    return not_taken();
  }
}
PyObject* py_gemv(PyObject*, PyObject* const* a, Py_ssize_t n) { return projection(a, n, false); }
PyObject* py_batch(PyObject*, PyObject* const* a, Py_ssize_t n) { return projection(a, n, true); }

// multi([(linear, x, y), ...])
PyObject* py_multi(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 1 || !g_multi || !(PyList_CheckExact(a[0]) || PyTuple_CheckExact(a[0]))) return not_taken();
  const Py_ssize_t count = PySequence_Fast_GET_SIZE(a[0]);
  if (count < 1 || count > CUDALM_B200_MAX_INLINE_LINEARS) return not_taken();
  try {
    const int dev = c10::cuda::current_device();
    cudalm_b200_linear ls[CUDALM_B200_MAX_INLINE_LINEARS];
    for (Py_ssize_t i = 0; i < count; ++i) {
      PyObject* item = PySequence_Fast_GET_ITEM(a[0], i);
      if (!PyTuple_CheckExact(item) || PyTuple_GET_SIZE(item) != 3) return not_taken();
      Lin lin;
      const at::Tensor* x = plain(PyTuple_GET_ITEM(item, 1), at::kBFloat16, dev);
      const at::Tensor* y = plain(PyTuple_GET_ITEM(item, 2), at::kBFloat16, dev);
      if (!x || !y || !read_linear(PyTuple_GET_ITEM(item, 0), dev, &lin)) return not_taken();
      const int64_t M = rows_of(*x);
      if (M < 1 || M > kIntMax || x->numel() != M * lin.K || y->numel() != M * lin.N) return not_taken();
      ls[i] = cudalm_b200_linear{bytes(lin.weight), halves(lin.scale), halves(x), halves(y),
                                 static_cast<int32_t>(lin.N), static_cast<int32_t>(lin.K),
                                 static_cast<int32_t>(M), 0};
    }
    void* st = stream_of(dev);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_multi(ls, static_cast<int>(count), st);
    Py_END_ALLOW_THREADS
    return status(rc);
  } catch (...) {
    return not_taken();
  }
}

// gate_up_silu(gate, up, x, out)
PyObject* py_gate_up_silu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4 || !g_gate_up_silu) return not_taken();
  try {
    const int dev = c10::cuda::current_device();
    Lin g, u;
    const at::Tensor* x = plain(a[2], at::kBFloat16, dev);
    const at::Tensor* y = plain(a[3], at::kBFloat16, dev);
    if (!x || !y || !read_linear(a[0], dev, &g) || !read_linear(a[1], dev, &u)) return not_taken();
    const int64_t M = rows_of(*x);
    if (g.N != u.N || g.K != u.K || M < 1 || M > kIntMax || x->numel() != M * g.K || y->numel() < M * g.N)
      return not_taken();
    const uint8_t *gw = bytes(g.weight), *uw = bytes(u.weight);
    uint16_t *gs = halves(g.scale), *us = halves(u.scale), *xp = halves(x), *yp = halves(y);
    void* st = stream_of(dev);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_gate_up_silu(gw, gs, uw, us, xp, yp, static_cast<int>(g.N), static_cast<int>(g.K),
                        static_cast<int>(M), st);
    Py_END_ALLOW_THREADS
    return status(rc);
  } catch (...) {
    return not_taken();
  }
}

// linear_residual(linear, x, residual, y)
PyObject* py_residual(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4 || !g_residual) return not_taken();
  try {
    const int dev = c10::cuda::current_device();
    Lin l;
    const at::Tensor* x = plain(a[1], at::kBFloat16, dev);
    const at::Tensor* r = plain(a[2], at::kBFloat16, dev);
    const at::Tensor* y = plain(a[3], at::kBFloat16, dev);
    if (!x || !r || !y || !read_linear(a[0], dev, &l)) return not_taken();
    const int64_t M = rows_of(*x);
    if (M < 1 || M > kIntMax || x->numel() != M * l.K || r->numel() < M * l.N || y->numel() < M * l.N)
      return not_taken();
    const uint8_t* wp = bytes(l.weight);
    uint16_t *sp = halves(l.scale), *xp = halves(x), *rp = halves(r), *yp = halves(y);
    void* st = stream_of(dev);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = g_residual(wp, sp, xp, rp, yp, static_cast<int>(l.N), static_cast<int>(l.K), static_cast<int>(M), st);
    Py_END_ALLOW_THREADS
    return status(rc);
  } catch (...) {
    return not_taken();
  }
}

// bind(gemv, batch, multi, gate_up_silu, linear_residual): entry point addresses
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "bind takes five addresses");
    return nullptr;
  }
  void* p[5];
  for (int i = 0; i < 5; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i]) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
      return nullptr;
    }
  }
  g_gemv = reinterpret_cast<decltype(g_gemv)>(p[0]);
  g_batch = reinterpret_cast<decltype(g_batch)>(p[1]);
  g_multi = reinterpret_cast<decltype(g_multi)>(p[2]);
  g_gate_up_silu = reinterpret_cast<decltype(g_gate_up_silu)>(p[3]);
  g_residual = reinterpret_cast<decltype(g_residual)>(p[4]);
  Py_RETURN_NONE;
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  static PyMethodDef methods[] = {
      {"bind", fast(py_bind), METH_FASTCALL, nullptr},
      {"gemv", fast(py_gemv), METH_FASTCALL, nullptr},
      {"batch", fast(py_batch), METH_FASTCALL, nullptr},
      {"multi", fast(py_multi), METH_FASTCALL, nullptr},
      {"gate_up_silu", fast(py_gate_up_silu), METH_FASTCALL, nullptr},
      {"linear_residual", fast(py_residual), METH_FASTCALL, nullptr},
      {nullptr, nullptr, 0, nullptr}};
  static PyModuleDef def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods,
                            nullptr,               nullptr,   nullptr, nullptr};
  s_weight = PyUnicode_InternFromString("weight");
  s_scale = PyUnicode_InternFromString("scale");
  s_N = PyUnicode_InternFromString("N");
  s_K = PyUnicode_InternFromString("K");
  return PyModule_Create(&def);
}
