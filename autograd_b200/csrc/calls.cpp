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

PyObject *s_storage, *s_ptr, *s_buffer_id, *s_offset, *s_shape;

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
    if constexpr (std::is_same_v<R, size_t>) {
      return PyLong_FromSize_t(r);
    } else {
      if (r == AG_OK) Py_RETURN_NONE;
      const char* msg = ag_last_error(std::get<0>(a));
      PyObject* e = PyObject_CallFunction(g_error, "is", (int)r, msg ? msg : "");
      if (e) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
      }
      return nullptr;
    }
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
  g_error = PyExc_RuntimeError;
  Py_INCREF(g_error);
  return m;
}
