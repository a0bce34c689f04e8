// CPython module `_calls`: the entry points that a step calls hundreds of times, each as one
// METH_FASTCALL function that converts its arguments, calls the C function without the GIL and raises
// AgError on a non-zero status.
//
// What bounds a step of small kernels is the host: a ctypes call with a dozen pointer and size arguments
// builds a dozen Python objects and costs 2.5-3.5 us, more than the launch it makes; here the conversion is
// a few compares per argument (0.2-0.3 us per call): the 82 launches of one generated token (20 layers, hidden
// 1280, 8 sequences) took 320 us instead of 457 through ctypes, with the same kernels.
// Argument rules are those of context.py: an address is an int or None (NULL), or the tensor or storage that has
// it; sizes and flags are anything with __int__, the CE descriptor is any object whose buffer is an ag_flce_desc.
// Everything that is not called per launch stays with the binding of _native.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>
#include <cstdint>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "autograd_b200.h"

namespace {

PyObject* g_error = nullptr;  // autograd_b200._native.AgError

// value of an int-like object; sets a Python error and returns 0 on failure
long long as_int(PyObject* o) {
  if (PyLong_Check(o)) return PyLong_AsLongLong(o);
  PyObject* n = PyNumber_Long(o);
  if (!n) return 0;
  const long long v = PyLong_AsLongLong(n);
  Py_DECREF(n);
  return v;
}

PyObject *s_storage, *s_ptr, *s_buffer_id, *s_offset, *s_shape, *s_dtype, *s_hi;

// address of a storage: its memory pointer's base and offset
void* storage_address(PyObject* st) {
  PyObject* p = PyObject_GetAttr(st, s_ptr);
  if (!p) return nullptr;
  PyObject *b = PyObject_GetAttr(p, s_buffer_id), *o = b ? PyObject_GetAttr(p, s_offset) : nullptr;
  Py_DECREF(p);
  void* at = o ? (char*)PyLong_AsVoidPtr(b) + PyLong_AsSsize_t(o) : nullptr;
  Py_XDECREF(b);
  Py_XDECREF(o);
  return at;
}

// An address is an int, None (NULL), a tensor-like object with a storage (None: NULL), or a storage itself.  The type
// of the last storage seen is remembered, which spares its kind the failing look for `.storage`.
void* as_address(PyObject* o) {
  static PyTypeObject* storage_type = nullptr;
  if (o == Py_None) return nullptr;
  if (PyLong_Check(o)) return PyLong_AsVoidPtr(o);
  if (Py_TYPE(o) == storage_type) return storage_address(o);
  PyObject* st = PyObject_GetAttr(o, s_storage);
  if (st) {
    void* at = st == Py_None ? nullptr : storage_address(st);
    Py_DECREF(st);
    return at;
  }
  if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return nullptr;
  PyErr_Clear();
  if (PyObject_HasAttr(o, s_ptr)) {
    Py_INCREF(Py_TYPE(o));
    Py_XSETREF(storage_type, Py_TYPE(o));
    return storage_address(o);
  }
  PyObject* n = PyNumber_Long(o);
  if (!n) return nullptr;
  void* p = PyLong_AsVoidPtr(n);
  Py_DECREF(n);
  return p;
}

template <typename T>
bool convert(PyObject* o, T& out) {
  if constexpr (std::is_same_v<T, const ag_flce_desc*>) {
    Py_buffer b;
    if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) return false;
    const bool fits = b.len == (Py_ssize_t)sizeof(ag_flce_desc);
    out = static_cast<const ag_flce_desc*>(b.buf);  // the caller's argument keeps the object alive
    PyBuffer_Release(&b);
    if (!fits) PyErr_SetString(PyExc_TypeError, "not an ag_flce_desc");
    return fits;
  } else if constexpr (std::is_pointer_v<T>) {
    void* p = as_address(o);
    if (!p && PyErr_Occurred()) return false;
    out = static_cast<T>(p);
    return true;
  } else if constexpr (std::is_floating_point_v<T>) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return false;
    out = static_cast<T>(v);
    return true;
  } else {
    const long long v = as_int(o);
    if (PyErr_Occurred()) return false;
    if constexpr (sizeof(T) == 4) {
      const bool fits = std::is_signed_v<T> ? (v >= INT_MIN && v <= INT_MAX) : (v >= 0 && v <= (long long)UINT_MAX);
      if (!fits) {
        PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits");
        return false;
      }
    }
    out = static_cast<T>(v);
    return true;
  }
}

// None, or the error that a status means
PyObject* checked(int status, ag_ctx* ctx) {
  if (status == AG_OK) Py_RETURN_NONE;
  const char* msg = ag_last_error(ctx);
  PyObject* e = PyObject_CallFunction(g_error, "is", status, msg ? msg : "");
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  return nullptr;
}

template <auto Fn, typename Sig>
struct Call;

template <auto Fn, typename R, typename... A>
struct Call<Fn, R (*)(A...)> {
  static PyObject* run(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != (Py_ssize_t)sizeof...(A)) {
      PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", (Py_ssize_t)sizeof...(A), n);
      return nullptr;
    }
    return go(args, std::index_sequence_for<A...>{});
  }
  template <size_t... I>
  static PyObject* go(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> a;
    if (!(convert(args[I], std::get<I>(a)) && ...)) return nullptr;
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = Fn(std::get<I>(a)...);
    Py_END_ALLOW_THREADS
    if constexpr (std::is_same_v<R, size_t>)
      return PyLong_FromSize_t(r);
    else
      return checked(r, std::get<0>(a));
  }
};

PyObject* set_error(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XSETREF(g_error, cls);
  Py_RETURN_NONE;
}

// What every kernel callable asks of its tensors, without a Python frame each: a dozen per call made a third of the
// backend layer's time.
PyObject* addr(PyObject*, PyObject* t) {
  void* at = as_address(t);
  if (!at && PyErr_Occurred()) return nullptr;
  return PyLong_FromVoidPtr(at);
}

// rows: product of the leading extents; cols: the last extent, -1 without one
bool extents(PyObject* t, long long& rows, long long& cols) {
  PyObject* shape = PyObject_GetAttr(t, s_shape);
  if (!shape) return false;
  PyObject* fast = PySequence_Fast(shape, "shape is not a sequence");
  Py_DECREF(shape);
  if (!fast) return false;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
  rows = 1;
  cols = -1;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const long long v = as_int(PySequence_Fast_GET_ITEM(fast, i));
    if (i + 1 < n) rows *= v; else cols = v;
  }
  Py_DECREF(fast);
  return !PyErr_Occurred();
}

PyObject* rows_cols(PyObject*, PyObject* t) {
  long long rows, cols;
  if (!extents(t, rows, cols)) return nullptr;
  if (cols < 0) {
    PyErr_SetString(PyExc_IndexError, "a scalar has no columns");
    return nullptr;
  }
  return Py_BuildValue("LL", rows, cols);
}

PyObject* size(PyObject*, PyObject* t) {
  long long rows, cols;
  if (!extents(t, rows, cols)) return nullptr;
  return PyLong_FromLongLong(cols < 0 ? 1 : rows * cols);
}

// ---------------------------------------------------------------------------- layer calls
// What a backend's callable does for one launch, in one call: the handle of its context, the extents and storage types of its
// tensors, the launch.  In Python that took two more frames and a tuple, 0.3 of 2.5 us of a call.  The forms in Python
// (`plain`, set by set_layers) remain for any other context than a CudaContext, for one whose method was replaced, on the
// class or on the object (a tracer, a timer), and for any other storage type than the two type objects that tensors usually
// carry.
PyObject *g_plain = nullptr, *g_context = nullptr, *g_f32 = nullptr, *g_bf16 = nullptr;

// The methods that the compiled forms stand in for, as they were when the layers were set up
enum { GELU_FORWARD, GELU_BACKWARD, ADD_LAYERNORM_FORWARD, RMSNORM_FORWARD, SWIGLU_FORWARD, SWIGLU_BACKWARD, ROPE_QK, FILL_F32,
       ADAMW_STEP, METHODS };
constexpr const char* kMethods[METHODS] = {"gelu_forward", "gelu_backward", "add_layernorm_forward", "rmsnorm_forward",
                                           "swiglu_forward", "swiglu_backward", "rope_qk", "fill_f32", "adamw_step"};
struct Method {
  PyObject *name, *function;
} g_method[METHODS];

PyObject* set_layers(PyObject*, PyObject* args) {
  PyObject *plain, *context, *f32, *bf16;
  if (!PyArg_ParseTuple(args, "OO!OO", &plain, &PyType_Type, &context, &f32, &bf16)) return nullptr;
  for (int i = 0; i < METHODS; ++i) {
    PyObject* name = PyUnicode_InternFromString(kMethods[i]);
    if (!name) return nullptr;
    Py_XSETREF(g_method[i].name, name);
    PyObject* f = PyDict_GetItemWithError(reinterpret_cast<PyTypeObject*>(context)->tp_dict, name);
    if (!f && PyErr_Occurred()) return nullptr;
    Py_XINCREF(f);  // absent: the form in Python is always taken
    Py_XSETREF(g_method[i].function, f);
  }
  for (PyObject* o : {plain, context, f32, bf16}) Py_INCREF(o);
  Py_XSETREF(g_plain, plain);
  Py_XSETREF(g_context, context);
  Py_XSETREF(g_f32, f32);
  Py_XSETREF(g_bf16, bf16);
  Py_RETURN_NONE;
}

// AG_F32 or AG_BF16 of a storage; -1: some other object for it
int storage_dtype(PyObject* st) {
  PyObject* d = PyObject_GetAttr(st, s_dtype);
  if (!d) {
    PyErr_Clear();
    return -1;
  }
  const int r = d == g_f32 ? AG_F32 : d == g_bf16 ? AG_BF16 : -1;
  Py_DECREF(d);
  return r;
}
int tensor_dtype(PyObject* t) {
  PyObject* st = PyObject_GetAttr(t, s_storage);
  if (!st) {
    PyErr_Clear();
    return -1;
  }
  const int r = storage_dtype(st);
  Py_DECREF(st);
  return r;
}

struct Layer {
  PyObject* const* args;
  Py_ssize_t n;
  ag_ctx* ctx = nullptr;
  bool ok = true;  // no Python error so far

  // Whether the compiled form applies; otherwise go on with plain()
  bool real(int method) {
    const Method& m = g_method[method];
    PyTypeObject* type = Py_TYPE(args[0]);
    if ((PyObject*)type != g_context || PyDict_GetItemWithError(type->tp_dict, m.name) != m.function || !m.function) return false;
    PyObject* own = PyObject_GenericGetDict(args[0], nullptr);
    PyObject* h = own && !PyDict_GetItemWithError(own, m.name) ? PyDict_GetItemWithError(own, s_hi) : nullptr;
    if (h) ctx = static_cast<ag_ctx*>(PyLong_AsVoidPtr(h));
    Py_XDECREF(own);  // the context keeps it
    if (!h) PyErr_Clear();
    else if (!ctx && PyErr_Occurred()) ok = false;
    return h != nullptr;
  }
  PyObject* plain(const char* name) {
    PyObject* f = g_plain ? PyObject_GetAttrString(g_plain, name) : nullptr;
    if (!f) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "layer calls are not set up");
      return nullptr;
    }
    PyObject* r = PyObject_Vectorcall(f, args, (size_t)n, nullptr);
    Py_DECREF(f);
    return r;
  }
  template <typename T = float>
  T* at(int i) {
    T* p = nullptr;
    if (ok) ok = convert(args[i], p);
    return p;
  }
  double number(int i) {
    double v = 0.0;
    if (ok) ok = convert(args[i], v);
    return v;
  }
  // a row of `parts` times what has to fit 32 bits
  void rows_cols(int i, long long& rows, long long& cols, int parts = 1) {
    rows = cols = 0;
    if (!ok) return;
    ok = extents(args[i], rows, cols);
    if (ok && cols < 0) {
      PyErr_SetString(PyExc_IndexError, "a scalar has no columns");
      ok = false;
    }
    if (ok && cols / parts > INT_MAX) {
      PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits");
      ok = false;
    }
  }
  long long size(int i) {
    long long rows = 0, cols = 0;
    if (ok) ok = extents(args[i], rows, cols);
    return cols < 0 ? 1 : rows * cols;
  }
  template <typename F>
  PyObject* launch(F&& f) {
    if (!ok) return nullptr;
    int r;
    Py_BEGIN_ALLOW_THREADS
    r = f();
    Py_END_ALLOW_THREADS
    return checked(r, ctx);
  }
};

#define LAYER(name, count)                                                                                   \
  PyObject* layer_##name##_run(Layer l);                                                                     \
  PyObject* layer_##name(PyObject*, PyObject* const* args, Py_ssize_t n) {                                   \
    if (n != count) {                                                                                        \
      PyErr_Format(PyExc_TypeError, "%d arguments expected, got %zd", count, n);                             \
      return nullptr;                                                                                        \
    }                                                                                                        \
    return layer_##name##_run(Layer{args, n});                                                               \
  }                                                                                                          \
  PyObject* layer_##name##_run(Layer l)

LAYER(gelu_forward, 3) {  // ctx, x, y
  if (!l.real(GELU_FORWARD)) return l.plain("gelu_forward");
  float *x = l.at(1), *y = l.at(2);
  const long long n = l.size(1);
  return l.launch([&] { return ag_gelu_forward(l.ctx, x, y, n); });
}

LAYER(gelu_backward, 4) {  // ctx, x, dy, dx: dx += local
  if (!l.real(GELU_BACKWARD)) return l.plain("gelu_backward");
  float *x = l.at(1), *dy = l.at(2), *dx = l.at(3);
  const long long n = l.size(1);
  return l.launch([&] { return ag_gelu_backward(l.ctx, x, dy, dx, dx, n); });
}

LAYER(add_layernorm_forward, 10) {  // ctx, x, r, gamma, beta, h, y, mean, rstd, eps
  if (!l.real(ADD_LAYERNORM_FORWARD)) return l.plain("add_layernorm_forward");
  float *x = l.at(1), *r = l.at(2), *gamma = l.at(3), *beta = l.at(4), *h = l.at(5), *y = l.at(6), *mean = l.at(7), *rstd = l.at(8);
  const float eps = (float)l.number(9);
  long long rows, cols;
  l.rows_cols(1, rows, cols);
  return l.launch([&] { return ag_add_layernorm_forward(l.ctx, x, r, gamma, beta, h, y, mean, rstd, rows, (int)cols, eps); });
}

LAYER(rmsnorm_forward, 6) {  // ctx, x, gamma, y, inv_rms, eps
  const int dtype = tensor_dtype(l.args[1]);
  if (dtype < 0 || !l.real(RMSNORM_FORWARD)) return l.plain("rmsnorm_forward");
  void *x = l.at<void>(1), *y = l.at<void>(3);
  float *gamma = l.at(2), *inv_rms = l.at(4);
  const float eps = (float)l.number(5);
  long long rows, cols;
  l.rows_cols(1, rows, cols);
  return l.launch([&] { return ag_rmsnorm_forward(l.ctx, x, gamma, y, inv_rms, rows, (int)cols, eps, dtype); });
}

LAYER(swiglu_forward, 3) {  // ctx, gu, hidden
  const int dtype = tensor_dtype(l.args[1]);
  if (dtype < 0 || !l.real(SWIGLU_FORWARD)) return l.plain("swiglu_forward");
  void *gu = l.at<void>(1), *hidden = l.at<void>(2);
  long long rows, cols;
  l.rows_cols(1, rows, cols, 2);
  return l.launch([&] { return ag_swiglu_forward(l.ctx, gu, hidden, rows, (int)(cols / 2), dtype); });
}

LAYER(swiglu_backward, 3) {  // ctx, gu, dhidden
  const int dtype = tensor_dtype(l.args[1]);
  if (dtype < 0 || !l.real(SWIGLU_BACKWARD)) return l.plain("swiglu_backward");
  void *gu = l.at<void>(1), *dhidden = l.at<void>(2);
  long long rows, cols;
  l.rows_cols(1, rows, cols, 2);
  return l.launch([&] { return ag_swiglu_backward(l.ctx, gu, dhidden, rows, (int)(cols / 2), dtype); });
}

LAYER(rope_qk, 12) {  // ctx, q, k, cos, sin, b, t, h, hkv, d, sin_sign, dtype
  if (!l.real(ROPE_QK)) return l.plain("rope_qk");
  void *q = l.at<void>(1), *k = l.at<void>(2);
  float *cos = l.at(3), *sin = l.at(4);
  int v[7] = {};
  for (int i = 0; i < 7 && l.ok; ++i) l.ok = convert(l.args[5 + i], v[i]);
  return l.launch([&] {
    return ag_rope_qk(l.ctx, q, k, cos, sin, v[0], v[1], v[2], v[3], v[4], (int64_t)v[2] * v[4], (int64_t)v[3] * v[4], v[5], v[6]);
  });
}

LAYER(fill, 3) {  // ctx, storage, value
  const bool number = PyFloat_Check(l.args[2]) || PyLong_Check(l.args[2]);  // the form in Python also takes text, as float() does
  if (!number || storage_dtype(l.args[1]) != AG_F32 || !l.real(FILL_F32)) return l.plain("fill");
  float* dst = l.at(1);
  const float value = (float)l.number(2);
  const long long n = l.size(1);
  return l.launch([&] { return ag_fill_f32(l.ctx, dst, value, n); });
}

LAYER(adamw_step, 12) {  // ctx, p, g, m, v, lr, lr_t, b1, b2, eps, weight_decay, grad_scale
  const int dtype = storage_dtype(l.args[2]);
  if (dtype < 0 || !l.real(ADAMW_STEP)) return l.plain("adamw_step");
  float *p = l.at(1), *m = l.at(3), *v = l.at(4);
  void* g = l.at<void>(2);
  double c[7];
  for (int i = 0; i < 7; ++i) c[i] = l.number(5 + i);
  const long long n = l.size(1);
  return l.launch([&] {
    return dtype == AG_BF16
               ? ag_adamw_step_bf16grad(l.ctx, p, (const uint16_t*)g, m, v, n, c[0], c[1], c[2], c[3], c[4], c[5], c[6])
               : ag_adamw_step(l.ctx, p, (const float*)g, m, v, n, c[0], c[1], c[2], c[3], c[4], c[5], c[6]);
  });
}

#define LAYER_METHOD(name) {"layer_" #name, (PyCFunction)(void (*)(void))layer_##name, METH_FASTCALL, nullptr}
#define CALL(name) {#name, (PyCFunction)(void (*)(void))Call<&name, decltype(&name)>::run, METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    {"set_error", set_error, METH_O, "class raised on a non-zero status, called with (code, message)"},
    CALL(ag_fill_f32),
    CALL(ag_fill_pattern),
    CALL(ag_add_forward),
    CALL(ag_add_backward),
    CALL(ag_add_layernorm_forward),
    CALL(ag_norm_partials_bytes),
    CALL(ag_layernorm_backward),
    CALL(ag_layernorm_backward_noalloc),
    CALL(ag_rmsnorm_forward),
    CALL(ag_rmsnorm_backward),
    CALL(ag_gelu_forward),
    CALL(ag_gelu_backward),
    CALL(ag_swiglu_forward),
    CALL(ag_swiglu_backward),
    CALL(ag_rope_qk),
    CALL(ag_gather_forward),
    CALL(ag_gather_backward),
    CALL(ag_gather_backward_bf16),
    CALL(ag_f32_to_bf16),
    CALL(ag_bf16_to_f32),
    CALL(ag_scatter_add_scratch_bytes),
    CALL(ag_flce_scratch_bytes),
    CALL(ag_linear_add_scratch_bytes),
    CALL(ag_flce_forward),
    CALL(ag_flce_backward),
    CALL(ag_flce_logits_bytes),
    CALL(ag_zero_ranges),
    CALL(ag_layernorm_backward_rows),
    CALL(ag_norm_partials_add),
    CALL(ag_flce_forward_keep),
    CALL(ag_flce_backward_kept),
    CALL(ag_linear_add_forward),
    CALL(ag_linear_add_backward),
    CALL(ag_adamw_step),
    CALL(ag_adamw_step_bf16grad),
    CALL(ag_event_record),
    CALL(ag_graph_launch),
    {"addr", addr, METH_O, "device address of a tensor-like object or a storage: 0 for None or without storage"},
    {"size", size, METH_O, "number of elements of anything with a shape"},
    {"rows_cols", rows_cols, METH_O, "(product of the leading extents, last extent) of a tensor-like object"},
    CALL(ag_copy_h2d),
    {"set_layers", set_layers, METH_VARARGS, "(forms in Python, context class, type objects of fp32 and bf16 storages)"},
    LAYER_METHOD(gelu_forward),
    LAYER_METHOD(gelu_backward),
    LAYER_METHOD(add_layernorm_forward),
    LAYER_METHOD(rmsnorm_forward),
    LAYER_METHOD(swiglu_forward),
    LAYER_METHOD(swiglu_backward),
    LAYER_METHOD(rope_qk),
    LAYER_METHOD(fill),
    LAYER_METHOD(adamw_step),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", "launch entry points of libautograd_b200.so", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  PyObject* m = PyModule_Create(&module);
  if (!m) return nullptr;
  s_storage = PyUnicode_InternFromString("storage");
  s_ptr = PyUnicode_InternFromString("ptr");
  s_buffer_id = PyUnicode_InternFromString("buffer_id");
  s_offset = PyUnicode_InternFromString("offset");
  s_shape = PyUnicode_InternFromString("shape");
  s_dtype = PyUnicode_InternFromString("dtype");
  s_hi = PyUnicode_InternFromString("_hi");
  g_error = PyExc_RuntimeError;
  Py_INCREF(g_error);
  return m;
}
