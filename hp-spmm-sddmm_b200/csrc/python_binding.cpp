// CPython face of the calls a program makes once per product: argument conversion in C.
//
// A product on a small matrix takes the GPU a few microseconds, and through ctypes the conversion of its
// thirteen arguments, together with the Python code that prepares them, took as long.  The functions here take
// what the Python layer is given and call the C ABI, with the interpreter lock released.  They return the status code.
// What they accept is what ctypes accepts for the same call:
//   buffers    None, a numpy array, a DeviceBuffer, or whatever int() takes
//   handles    (context, plan, layer, stream) None, an integer, a ctypes pointer, an object with _as_parameter_
//   integers   an integer (cut to 64 bits), a ctypes integer, an object with __index__ or _as_parameter_
//   options    a false value for none, or an Opts structure
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "hpspmm.h"

namespace {

// addresses of the C ABI in the library the package has loaded (bind)
struct {
  decltype(&hpspmm_spmm_csr_f32) spmm_csr;
  decltype(&hpspmm_spmm_coo_f32) spmm_coo;
  decltype(&hpspmm_sddmm_csr_f32) sddmm_csr;
  decltype(&hpspmm_fill_f32) fill;
  decltype(&hpspmm_layer_forward) layer_forward;
  decltype(&hpspmm_layer_backward_features) layer_backward_features;
  decltype(&hpspmm_layer_backward_weights) layer_backward_weights;
} api;

PyObject *s_ptr, *s_value, *s_ctypes, *s_data, *s_as_parameter;
PyObject *t_ndarray, *t_buffer, *t_opts;   // numpy.ndarray, DeviceBuffer, Opts (bind)

// 64 bits of a Python integer, higher ones cut off as ctypes does
bool low_bits(PyObject* v, uint64_t* out) {
  *out = PyLong_AsUnsignedLongLongMask(v);
  return !(*out == (uint64_t)-1 && PyErr_Occurred());
}

bool as_address(PyObject* o, void** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  uint64_t bits = 0;
  bool ok;
  if (PyLong_Check(o)) {
    ok = low_bits(o, &bits);
  } else {
    PyObject* v = nullptr;
    int is = PyObject_IsInstance(o, t_ndarray);
    if (is < 0) return false;
    if (is) {
      PyObject* c = PyObject_GetAttr(o, s_ctypes);
      if (c) {
        v = PyObject_GetAttr(c, s_data);
        Py_DECREF(c);
      }
    } else {
      is = PyObject_IsInstance(o, t_buffer);
      if (is < 0) return false;
      v = is ? PyObject_GetAttr(o, s_ptr) : PyNumber_Long(o);
    }
    if (!v) return false;
    ok = v == Py_None || low_bits(v, &bits);
    Py_DECREF(v);
  }
  *out = (void*)(uintptr_t)bits;
  return ok;
}

// the integer behind a handle or size: itself, the `value` of a ctypes object, what _as_parameter_ leads to.  A new
// reference, None for a null pointer.
PyObject* plain_integer(PyObject* o, int depth = 0) {
  if (o == Py_None || PyLong_Check(o)) return Py_NewRef(o);
  PyObject* v = PyObject_GetAttr(o, s_value);
  if (!v) {
    PyErr_Clear();
    v = PyObject_GetAttr(o, s_as_parameter);
  }
  if (!v) {
    PyErr_Clear();
    return PyNumber_Index(o);
  }
  PyObject* r = depth < 4 ? plain_integer(v, depth + 1) : nullptr;
  if (!r && !PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "_as_parameter_ leads to no integer");
  Py_DECREF(v);
  return r;
}

bool as_handle(PyObject* o, void** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  PyObject* v = plain_integer(o);
  if (!v) return false;
  uint64_t bits = 0;
  const bool ok = v == Py_None || low_bits(v, &bits);
  Py_DECREF(v);
  *out = (void*)(uintptr_t)bits;
  return ok;
}

bool as_int(PyObject* o, int64_t* out) {
  *out = 0;
  PyObject* v = plain_integer(o);
  if (!v) return false;
  uint64_t bits = 0;
  bool ok = false;
  if (PyLong_Check(v))
    ok = low_bits(v, &bits);
  else
    PyErr_SetString(PyExc_TypeError, "an integer is required");
  Py_DECREF(v);
  *out = (int64_t)bits;
  return ok;
}

bool as_opts(PyObject* o, hpspmm_opts* buf, const hpspmm_opts** out) {
  *out = nullptr;
  if (o == Py_None) return true;
  const int given = PyObject_IsTrue(o);
  if (given < 0) return false;
  if (!given) return true;
  const int is = PyObject_IsInstance(o, t_opts);
  if (is < 0) return false;
  if (!is) {
    PyErr_SetString(PyExc_TypeError, "opts must be an Opts structure");
    return false;
  }
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) != 0) return false;
  memcpy(buf, view.buf, sizeof(*buf));   // (a subclass may add fields behind them)
  *out = buf;
  PyBuffer_Release(&view);
  return true;
}

// converts args[0 .. n): a buffer where `kinds` has 'p', a handle where it has 'h', an integer where it has 'i'
bool convert(PyObject* const* args, const char* kinds, void** p, int64_t* v) {
  for (int i = 0; kinds[i]; ++i)
    if (kinds[i] == 'p' ? !as_address(args[i], p + i) : kinds[i] == 'h' ? !as_handle(args[i], p + i) : !as_int(args[i], v + i))
      return false;
  return true;
}

bool arity(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, n);
  return false;
}

// ctx, plan, M, N, K, nnz, row_ptr, col_idx, vals | X, B | Y, C | out, opts, stream
template <typename F>
PyObject* csr_call(F fn, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 13)) return nullptr;
  void* p[13];
  int64_t v[13];
  hpspmm_opts buf;
  const hpspmm_opts* opts;
  if (!convert(a, "hhiiiippppp", p, v) || !as_opts(a[11], &buf, &opts) || !as_handle(a[12], &p[12])) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = fn((hpspmm_ctx*)p[0], (const hpspmm_plan*)p[1], v[2], v[3], v[4], v[5], (const int32_t*)p[6],
          (const int32_t*)p[7], (const float*)p[8], (const float*)p[9], (float*)p[10], opts, p[12]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

PyObject* py_spmm_csr(PyObject*, PyObject* const* a, Py_ssize_t n) { return csr_call(api.spmm_csr, a, n); }
PyObject* py_sddmm_csr(PyObject*, PyObject* const* a, Py_ssize_t n) { return csr_call(api.sddmm_csr, a, n); }

// ctx, M, N, K, nnz_padded, row_idx, col_idx, vals, B, C, opts, stream
PyObject* py_spmm_coo(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 12)) return nullptr;
  void* p[12];
  int64_t v[12];
  hpspmm_opts buf;
  const hpspmm_opts* opts;
  if (!convert(a, "hiiiippppp", p, v) || !as_opts(a[10], &buf, &opts) || !as_handle(a[11], &p[11])) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = api.spmm_coo((hpspmm_ctx*)p[0], v[1], v[2], v[3], v[4], (const int32_t*)p[5], (const int32_t*)p[6],
                    (const float*)p[7], (const float*)p[8], (float*)p[9], opts, p[11]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// ctx, dev, count, value, stream
PyObject* py_fill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 5)) return nullptr;
  void *ctx, *dev, *stream;
  int64_t count;
  if (!as_handle(a[0], &ctx) || !as_address(a[1], &dev) || !as_int(a[2], &count) || !as_handle(a[4], &stream))
    return nullptr;
  const double value = PyFloat_AsDouble(a[3]);
  if (value == -1.0 && PyErr_Occurred()) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = api.fill((hpspmm_ctx*)ctx, (float*)dev, count, (float)value, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// ctx, layer, K, in, out, stream
template <typename F>
PyObject* layer_call(F fn, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 6)) return nullptr;
  void* p[6];
  int64_t v[6];
  if (!convert(a, "hhipph", p, v)) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = fn((hpspmm_ctx*)p[0], (hpspmm_layer*)p[1], v[2], (const float*)p[3], (float*)p[4], p[5]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

PyObject* py_layer_forward(PyObject*, PyObject* const* a, Py_ssize_t n) { return layer_call(api.layer_forward, a, n); }
PyObject* py_layer_backward_features(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return layer_call(api.layer_backward_features, a, n);
}

// ctx, layer, K, dC, H, dA, stream
PyObject* py_layer_backward_weights(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 7)) return nullptr;
  void* p[7];
  int64_t v[7];
  if (!convert(a, "hhippph", p, v)) return nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = api.layer_backward_weights((hpspmm_ctx*)p[0], (hpspmm_layer*)p[1], v[2], (const float*)p[3], (const float*)p[4],
                                  (float*)p[5], p[6]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(st);
}

// bind(spmm_csr, spmm_coo, sddmm_csr, fill, layer_forward, layer_backward_features, layer_backward_weights, ndarray,
// DeviceBuffer, Opts): addresses in the loaded library, and the classes the arguments are tested for
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arity(n, 10)) return nullptr;
  void* p[7];
  int64_t unused[7];
  if (!convert(a, "hhhhhhh", p, unused)) return nullptr;
  PyObject** types[3] = {&t_ndarray, &t_buffer, &t_opts};
  for (int i = 0; i < 3; ++i) {
    PyObject* before = *types[i];
    *types[i] = Py_NewRef(a[7 + i]);
    Py_XDECREF(before);
  }
  api.spmm_csr = (decltype(api.spmm_csr))p[0];
  api.spmm_coo = (decltype(api.spmm_coo))p[1];
  api.sddmm_csr = (decltype(api.sddmm_csr))p[2];
  api.fill = (decltype(api.fill))p[3];
  api.layer_forward = (decltype(api.layer_forward))p[4];
  api.layer_backward_features = (decltype(api.layer_backward_features))p[5];
  api.layer_backward_weights = (decltype(api.layer_backward_weights))p[6];
  Py_RETURN_NONE;
}

#define FAST(name) \
  { #name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr }
PyMethodDef methods[] = {FAST(bind),          FAST(spmm_csr),      FAST(spmm_coo),
                         FAST(sddmm_csr),     FAST(fill),          FAST(layer_forward),
                         FAST(layer_backward_features), FAST(layer_backward_weights), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hpspmm_native", "Calls into libhpspmm.so", -1, methods,
                      nullptr,               nullptr,          nullptr,                   nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hpspmm_native(void) {
  s_ptr = PyUnicode_InternFromString("ptr");
  s_value = PyUnicode_InternFromString("value");
  s_ctypes = PyUnicode_InternFromString("ctypes");
  s_data = PyUnicode_InternFromString("data");
  s_as_parameter = PyUnicode_InternFromString("_as_parameter_");
  return PyModule_Create(&module);
}
