// CPython binding of the library's hot entry points on torch tensors.
//
// A call through ctypes costs 15 to 25 us of host time (tensor properties, broadcasts and allocations one Python call
// each, up to nineteen arguments to convert), more than most small calls run on the GPU.  Here the same work is done in
// C++: arguments that are what the library takes (CUDA tensors of the current device, contiguous, the right types) are
// passed on directly, outputs come from torch's caching allocator, the stream is the current one.  A function returns
// NotImplemented for anything else, and the Python wrapper of the same name converts the arguments and calls through
// ctypes.  The library's functions are handed over as addresses (init), so the binding links to no particular build.
// torch translates its own exceptions (HANDLE_TH_ERRORS): a declined allocation is a torch.OutOfMemoryError, as it is
// where the wrapper allocates.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>

#include "../../include/tallax_b200.h"

namespace {

struct Lib {
  decltype(&tlx_sample) sample;
  decltype(&tlx_sample_workspace_bytes) sample_workspace_bytes;
  decltype(&tlx_top_k) top_k;
  decltype(&tlx_top_k_workspace_bytes) top_k_workspace_bytes;
  decltype(&tlx_sort_carry) sort_carry;
  decltype(&tlx_sort_workspace_bytes) sort_workspace_bytes;
  decltype(&tlx_take_along_axis) take_along_axis;
  decltype(&tlx_cumsum) cumsum;
  decltype(&tlx_exchange_shard_candidates) exchange_shard_candidates;
  decltype(&tlx_exchange_merge_and_sample) exchange_merge_and_sample;
} lib;
PyObject* g_check = nullptr;   // Python: status code -> exception

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// The current device if `o` is a CUDA tensor on it, else -1.
int device_of(PyObject* o) {
  const at::Tensor* t = tensor(o);
  if (!t || !t->is_cuda()) return -1;
  const int dev = c10::cuda::current_device();
  return t->device().index() == dev ? dev : -1;
}
// A contiguous tensor on that device.
const at::Tensor* plain(PyObject* o, int device) {
  const at::Tensor* t = tensor(o);
  if (!t || !t->is_cuda() || t->device().index() != device || !t->is_contiguous()) return nullptr;
  return t;
}
const at::Tensor* plain(PyObject* o, int device, at::ScalarType type) {
  const at::Tensor* t = plain(o, device);
  return t && t->scalar_type() == type ? t : nullptr;
}
// One value per row.
const at::Tensor* vector(PyObject* o, int device, at::ScalarType type, int64_t rows) {
  const at::Tensor* t = plain(o, device, type);
  return t && t->dim() == 1 && t->size(0) == rows ? t : nullptr;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return TLX_F32;
    case at::kBFloat16: return TLX_BF16;
    case at::kHalf: return TLX_F16;
    case at::kInt: return TLX_I32;
    default: return -1;
  }
}

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, int device) {
  return at::detail::empty_cuda(size, type, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt);
}

bool finish(int rc) {
  if (rc == TLX_OK) return true;
  PyObject* r = PyObject_CallFunction(g_check, "i", rc);   // raises
  Py_XDECREF(r);
  if (r) PyErr_SetString(PyExc_RuntimeError, "tallax_b200: call failed");
  return false;
}

#define TLX_NOT_MINE Py_RETURN_NOTIMPLEMENTED

bool as_i64(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  *v = PyLong_AsLongLong(o);
  if (*v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
// Two words of a key given as a tuple or list of Python integers.
bool as_key(PyObject* o, uint32_t* k) {
  if (!PyTuple_CheckExact(o) && !PyList_CheckExact(o)) return false;
  if (PySequence_Fast_GET_SIZE(o) != 2) return false;
  for (int i = 0; i < 2; ++i) {
    int64_t v;
    if (!as_i64(PySequence_Fast_GET_ITEM(o, i), &v)) return false;
    k[i] = (uint32_t)v;
  }
  return true;
}

// sample(logits, top_k, top_p, temperature, rng_key, noise, dim0_offset) -> tokens
PyObject* py_sample(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor* x = plain(a[0], dev);
  if (!x || x->dim() != 2) TLX_NOT_MINE;
  const int64_t rows = x->size(0), vocab = x->size(1);
  const int dt = dtype_code(x->scalar_type());
  const at::Tensor* tk = vector(a[1], dev, at::kInt, rows);
  const at::Tensor* tp = vector(a[2], dev, at::kFloat, rows);
  const at::Tensor* te = vector(a[3], dev, at::kFloat, rows);
  uint32_t key[2] = {0, 0};
  const at::Tensor* noise = nullptr;
  int64_t offset;
  if (dt < 0 || !tk || !tp || !te || rows == 0 || vocab == 0 || !as_i64(a[6], &offset)) TLX_NOT_MINE;
  if (a[5] != Py_None) {
    noise = plain(a[5], dev, at::kFloat);
    if (!noise || noise->dim() != 2 || noise->size(1) < vocab) TLX_NOT_MINE;
  }
  if (a[4] != Py_None ? !as_key(a[4], key) : !noise) TLX_NOT_MINE;
  at::Tensor tokens = empty({rows}, at::kInt, dev);
  const size_t ws_bytes = lib.sample_workspace_bytes(rows, vocab);
  at::Tensor ws;
  if (ws_bytes > 256) ws = empty({(int64_t)ws_bytes}, at::kByte, dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.sample(st, x->data_ptr(), dt, rows, vocab, vocab, (const int32_t*)tk->data_ptr(), (const float*)tp->data_ptr(),
                  (const float*)te->data_ptr(), noise ? (const float*)noise->data_ptr() : nullptr, noise ? noise->size(1) : 0,
                  key[0], key[1], offset, (int32_t*)tokens.data_ptr(), nullptr, ws.defined() ? ws.data_ptr() : nullptr,
                  ws.defined() ? ws_bytes : 0);
  Py_END_ALLOW_THREADS
  return finish(rc) ? THPVariable_Wrap(tokens) : nullptr;
  END_HANDLE_TH_ERRORS
}

// top_k(x, k, k_per_row or None, replace_val or None) -> (values, indices), exact
PyObject* py_top_k(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor* x = plain(a[0], dev);
  int64_t k;
  if (!x || x->dim() != 2 || !as_i64(a[1], &k) || k < 1 || k > INT32_MAX) TLX_NOT_MINE;
  const int64_t rows = x->size(0), cols = x->size(1);
  const int dt = dtype_code(x->scalar_type());
  if (dt < 0) TLX_NOT_MINE;
  const at::Tensor* kpr = nullptr;
  double replace = 0.0;
  if (a[2] != Py_None && a[3] != Py_None) {
    kpr = vector(a[2], dev, at::kInt, rows);
    if (!kpr || !(PyFloat_CheckExact(a[3]) || PyLong_CheckExact(a[3]))) TLX_NOT_MINE;
    replace = PyFloat_AsDouble(a[3]);
    if (replace == -1.0 && PyErr_Occurred()) { PyErr_Clear(); TLX_NOT_MINE; }
  }
  at::Tensor vals = empty({rows, k}, x->scalar_type(), dev), idx = empty({rows, k}, at::kInt, dev), ws;
  // (floating-point rows need the workspace only beyond what a cluster holds)
  const size_t ws_bytes = dt == TLX_I32 || cols > 700000 ? lib.top_k_workspace_bytes(rows, cols, (int)k) : 0;
  if (ws_bytes) ws = empty({(int64_t)ws_bytes}, at::kByte, dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.top_k(st, x->data_ptr(), dt, rows, cols, cols, (int)k, kpr ? (const int32_t*)kpr->data_ptr() : nullptr, kpr != nullptr,
                 replace, 0, vals.data_ptr(), (int32_t*)idx.data_ptr(), nullptr, nullptr, nullptr,
                 ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? ws_bytes : 0);
  Py_END_ALLOW_THREADS
  if (!finish(rc)) return nullptr;
  PyObject* out = PyTuple_New(2);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(vals));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(idx));
  return out;
  END_HANDLE_TH_ERRORS
}

// argsort_rows(keys, descending, in_perm or None, want_keys, want_perm, carried, keys_among_them)
//   -> (keys or None, perm or None, *carried in the same order)
// carried: a tuple of tensors of the keys' shape, of which the first keys_among_them are further keys
PyObject* py_argsort_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor* x = plain(a[0], dev);
  if (!x || x->dim() != 2) TLX_NOT_MINE;
  const int64_t rows = x->size(0), cols = x->size(1);
  const int dt = dtype_code(x->scalar_type());
  auto same_shape = [&](const at::Tensor* t) { return t && t->dim() == 2 && t->size(0) == rows && t->size(1) == cols; };
  const at::Tensor* perm_in = nullptr;
  if (a[2] != Py_None) {
    perm_in = plain(a[2], dev, at::kInt);
    if (!same_shape(perm_in)) TLX_NOT_MINE;
  }
  const int desc = PyObject_IsTrue(a[1]), want_keys = PyObject_IsTrue(a[3]), want_perm = PyObject_IsTrue(a[4]);
  int64_t further;
  if (dt < 0 || desc < 0 || want_keys < 0 || want_perm < 0 || rows == 0 || cols == 0 || !PyTuple_CheckExact(a[5]) ||
      !as_i64(a[6], &further)) { PyErr_Clear(); TLX_NOT_MINE; }
  const Py_ssize_t count = PyTuple_GET_SIZE(a[5]);
  if (count > TLX_SORT_MAX_CARRIED) TLX_NOT_MINE;
  const at::Tensor* carried[TLX_SORT_MAX_CARRIED];
  for (Py_ssize_t i = 0; i < count; ++i) {
    carried[i] = plain(PyTuple_GET_ITEM(a[5], i), dev);
    if (!same_shape(carried[i]) || (carried[i]->element_size() != 2 && carried[i]->element_size() != 4)) TLX_NOT_MINE;
    if (i < further && dtype_code(carried[i]->scalar_type()) < 0) TLX_NOT_MINE;
  }
  at::Tensor keys, perm, ws, outs[TLX_SORT_MAX_CARRIED];
  tlx_sort_carried c[TLX_SORT_MAX_CARRIED];
  if (want_keys) keys = empty({rows, cols}, x->scalar_type(), dev);
  if (want_perm) perm = empty({rows, cols}, at::kInt, dev);
  for (Py_ssize_t i = 0; i < count; ++i) {
    outs[i] = empty({rows, cols}, carried[i]->scalar_type(), dev);
    c[i] = {carried[i]->data_ptr(), outs[i].data_ptr(), (int32_t)carried[i]->element_size(),
            i < further ? dtype_code(carried[i]->scalar_type()) : -1};
  }
  const size_t ws_bytes = cols > TLX_SORT_NO_WORKSPACE_N ? lib.sort_workspace_bytes(rows, cols) : 0;
  if (ws_bytes) ws = empty({(int64_t)ws_bytes}, at::kByte, dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.sort_carry(st, x->data_ptr(), dt, rows, cols, desc, perm_in ? (const int32_t*)perm_in->data_ptr() : nullptr,
                      want_keys ? keys.data_ptr() : nullptr, want_perm ? (int32_t*)perm.data_ptr() : nullptr, c, (int)count,
                      ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? ws_bytes : 0);
  Py_END_ALLOW_THREADS
  if (!finish(rc)) return nullptr;
  PyObject* out = PyTuple_New(2 + count);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, want_keys ? THPVariable_Wrap(keys) : Py_NewRef(Py_None));
  PyTuple_SET_ITEM(out, 1, want_perm ? THPVariable_Wrap(perm) : Py_NewRef(Py_None));
  for (Py_ssize_t i = 0; i < count; ++i) PyTuple_SET_ITEM(out, 2 + i, THPVariable_Wrap(outs[i]));
  return out;
  END_HANDLE_TH_ERRORS
}

// take_along_axis(values, indices, axis) -> out
PyObject* py_take_along_axis(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor *v = plain(a[0], dev), *i = plain(a[1], dev, at::kInt);
  int64_t axis;
  if (!v || !i || v->dim() != 2 || i->dim() != 2 || !as_i64(a[2], &axis) || axis < INT32_MIN || axis > INT32_MAX) TLX_NOT_MINE;
  at::Tensor out = empty(i->sizes(), v->scalar_type(), dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.take_along_axis(st, v->data_ptr(), (const int32_t*)i->data_ptr(), out.data_ptr(), v->size(0), v->size(1), i->size(0),
                           i->size(1), (int)v->element_size(), (int)axis);
  Py_END_ALLOW_THREADS
  return finish(rc) ? THPVariable_Wrap(out) : nullptr;
  END_HANDLE_TH_ERRORS
}

// cumsum(x, axis, reverse) -> out
PyObject* py_cumsum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor* x = plain(a[0], dev);
  int64_t axis;
  if (!x || x->dim() != 2 || !as_i64(a[1], &axis) || axis < INT32_MIN || axis > INT32_MAX) TLX_NOT_MINE;
  const int dt = dtype_code(x->scalar_type()), reverse = PyObject_IsTrue(a[2]);
  if (dt < 0 || reverse < 0) { PyErr_Clear(); TLX_NOT_MINE; }
  at::Tensor out = empty(x->sizes(), x->scalar_type(), dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.cumsum(st, x->data_ptr(), out.data_ptr(), x->size(0), x->size(1), dt, (int)axis, reverse);
  Py_END_ALLOW_THREADS
  return finish(rc) ? THPVariable_Wrap(out) : nullptr;
  END_HANDLE_TH_ERRORS
}

// exchange_step(logits_shard, col_offset, vocab_total, rng_key, noise_shard, dim0_offset, k_cand, rank, world, peers
// (address of the array of the ranks' buffers), own buffer, status, top_k, top_p, temperature, out or None) -> tokens
PyObject* py_exchange_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16) TLX_NOT_MINE;
  const int dev = device_of(a[0]);
  if (dev < 0) TLX_NOT_MINE;
  const at::Tensor* x = plain(a[0], dev);
  int64_t col0, vocab, offset, k, rank, world;
  if (!x || x->dim() != 2 || !as_i64(a[1], &col0) || !as_i64(a[2], &vocab) || !as_i64(a[5], &offset) || !as_i64(a[6], &k) ||
      !as_i64(a[7], &rank) || !as_i64(a[8], &world))
    TLX_NOT_MINE;
  const int64_t rows = x->size(0), v_local = x->size(1);
  const int dt = dtype_code(x->scalar_type());
  uint32_t key[2] = {0, 0};
  const at::Tensor* noise = nullptr;
  if (a[4] != Py_None) {
    noise = plain(a[4], dev, at::kFloat);
    if (!noise || noise->dim() != 2) TLX_NOT_MINE;
  }
  if (a[3] != Py_None ? !as_key(a[3], key) : !noise) TLX_NOT_MINE;
  const at::Tensor* status = plain(a[11], dev, at::kInt);
  const at::Tensor* tk = vector(a[12], dev, at::kInt, rows);
  const at::Tensor* tp = vector(a[13], dev, at::kFloat, rows);
  const at::Tensor* te = vector(a[14], dev, at::kFloat, rows);
  const at::Tensor* given = a[15] != Py_None ? vector(a[15], dev, at::kInt, rows) : nullptr;
  if (dt < 0 || !status || !tk || !tp || !te || (a[15] != Py_None && !given) || !PyLong_CheckExact(a[9]) || !PyLong_CheckExact(a[10]))
    TLX_NOT_MINE;
  void* peers = PyLong_AsVoidPtr(a[9]);
  void* own = PyLong_AsVoidPtr(a[10]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor tokens = given ? *given : empty({rows}, at::kInt, dev);
  void* st = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = lib.exchange_shard_candidates(st, x->data_ptr(), dt, rows, v_local, v_local, col0, (int)k,
                                     noise ? (const float*)noise->data_ptr() : nullptr, noise ? noise->size(1) : 0, nullptr, key[0],
                                     key[1], vocab, offset, nullptr, (int)rank, (int)world, (void* const*)peers);
  if (rc == TLX_OK)
    rc = lib.exchange_merge_and_sample(st, own, rows, (int)k, (int)world, (const int32_t*)tk->data_ptr(),
                                       (const float*)tp->data_ptr(), (const float*)te->data_ptr(), (int32_t*)tokens.data_ptr(),
                                       (int32_t*)status->data_ptr());
  Py_END_ALLOW_THREADS
  if (!finish(rc)) return nullptr;
  return given ? Py_NewRef(a[15]) : THPVariable_Wrap(tokens);
  END_HANDLE_TH_ERRORS
}

// init(check, {name: address})
PyObject* py_init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "init(check, addresses)");
    return nullptr;
  }
#define TLX_BIND(f)                                                        \
  {                                                                        \
    PyObject* v = PyDict_GetItemString(a[1], "tlx_" #f);                   \
    void* p = v ? PyLong_AsVoidPtr(v) : nullptr;                           \
    if (!p) {                                                              \
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "tlx_" #f);   \
      return nullptr;                                                      \
    }                                                                      \
    std::memcpy(&lib.f, &p, sizeof(p));                                    \
  }
  TLX_BIND(sample)
  TLX_BIND(sample_workspace_bytes)
  TLX_BIND(top_k)
  TLX_BIND(top_k_workspace_bytes)
  TLX_BIND(sort_carry)
  TLX_BIND(sort_workspace_bytes)
  TLX_BIND(take_along_axis)
  TLX_BIND(cumsum)
  TLX_BIND(exchange_shard_candidates)
  TLX_BIND(exchange_merge_and_sample)
  Py_INCREF(a[0]);
  Py_XDECREF(g_check);
  g_check = a[0];
  Py_RETURN_NONE;
}

#define TLX_METHOD(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {TLX_METHOD(init), TLX_METHOD(sample), TLX_METHOD(top_k), TLX_METHOD(argsort_rows),
                         TLX_METHOD(take_along_axis), TLX_METHOD(cumsum), TLX_METHOD(exchange_step), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tlx_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tlx_torch(void) { return PyModule_Create(&module); }
