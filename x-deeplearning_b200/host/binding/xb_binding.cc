// The calls of the Python binding that a serving loop makes many times a second, without ctypes: filling a structure field by
// field and converting every argument cost more than the launch behind it (gemm 4.9 us of Python, a feed 3.1 of which 1.0
// was the address of a NumPy array). No computation: the functions reach the C ABI through addresses that bind() is given, so
// that this module works on whichever libraries capi.py and blaze_api.py have loaded. Every C call runs without the
// interpreter lock, as ctypes does it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "xdlb200.h"

namespace {

struct Api {
  int (*gemm)(const xb_gemm_args*, xb_stream_t) = nullptr;
  int (*pool)(const xb_pool_group*, int32_t, void*, size_t, xb_stream_t) = nullptr;
  int (*reshape)(void*, const char*, const int*, int) = nullptr;
  int (*feed)(void*, const char*, void*, int) = nullptr;
} api;

PyObject *s_data_ptr, *s_dtype, *s_stride, *s_dim, *g_dtypes, *g_minus2;

// 0 and no exception, or -1 with one
int tensor_ptr(PyObject* t, void** out) {
  PyObject* r = PyObject_CallMethodNoArgs(t, s_data_ptr);
  if (!r) return -1;
  *out = PyLong_AsVoidPtr(r);
  Py_DECREF(r);
  return *out == nullptr && PyErr_Occurred() ? -1 : 0;
}
int tensor_dtype(PyObject* t, int32_t* out) {
  PyObject* d = PyObject_GetAttr(t, s_dtype);
  if (!d) return -1;
  PyObject* code = PyDict_GetItemWithError(g_dtypes, d);
  if (!code && !PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, d);
  Py_DECREF(d);
  if (!code) return -1;
  *out = (int32_t)PyLong_AsLong(code);
  return 0;
}
int as_i64(PyObject* v, int64_t* out) {
  *out = PyLong_AsLongLong(v);
  return *out == -1 && PyErr_Occurred() ? -1 : 0;
}
int as_i32(PyObject* v, int32_t* out) {
  const long x = PyLong_AsLong(v);
  if (x == -1 && PyErr_Occurred()) return -1;
  if (x < INT32_MIN || x > INT32_MAX) { PyErr_SetString(PyExc_OverflowError, "a size does not fit 32 bits"); return -1; }
  *out = (int32_t)x;
  return 0;
}
int as_flag(PyObject* v, int32_t* out) {
  const int x = PyObject_IsTrue(v);
  *out = x;
  return x < 0 ? -1 : 0;
}
int as_f32(PyObject* v, float* out) {
  const double x = PyFloat_AsDouble(v);
  *out = (float)x;
  return x == -1.0 && PyErr_Occurred() ? -1 : 0;
}
// a leading dimension: as given, or the tensor's stride of its last but one dimension
int leading(PyObject* given, PyObject* tensor, int64_t* out) {
  if (given != Py_None) return as_i64(given, out);
  PyObject* r = PyObject_CallMethodOneArg(tensor, s_stride, g_minus2);
  if (!r) return -1;
  const int rc = as_i64(r, out);
  Py_DECREF(r);
  return rc;
}

// gemm(A, B, Y, bias, trans_a, trans_b, alpha, beta, epilogue, ep, ep_count, nosqrt, engine, batch, strides, M, N, K, lda, ldb,
//      ldy, bias_kind, stride_ep, ldbias, bias_row_group, stream) -> xb_gemm's result. ops.gemm says what they are.
PyObject* py_gemm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  if (n != 26) { PyErr_SetString(PyExc_TypeError, "gemm: 26 arguments"); return nullptr; }
  xb_gemm_args a;
  memset(&a, 0, sizeof(a));
  void* p = nullptr;
  PyObject *A = v[0], *B = v[1], *Y = v[2], *bias = v[3], *ep = v[9], *strides = v[14];
  if (!PyTuple_Check(strides) || !PyTuple_Check(ep)) { PyErr_SetString(PyExc_TypeError, "gemm: strides and ep are tuples"); return nullptr; }
  if (PyTuple_GET_SIZE(strides) < 4 || PyTuple_GET_SIZE(ep) < 3) {
    PyErr_SetString(PyExc_IndexError, "gemm: four strides and three activation parameters");
    return nullptr;
  }
  auto st = [&](int i) { return PyTuple_GET_ITEM(strides, i); };
  if (as_i32(v[15], &a.M) || as_i32(v[16], &a.N) || as_i32(v[17], &a.K) || as_flag(v[4], &a.trans_a) || as_flag(v[5], &a.trans_b) ||
      as_f32(v[6], &a.alpha) || as_f32(v[7], &a.beta))
    return nullptr;
  if (tensor_ptr(A, &p) || leading(v[18], A, &a.lda) || as_i64(st(0), &a.stride_a)) return nullptr;
  a.A = p;
  if (tensor_ptr(B, &p) || leading(v[19], B, &a.ldb) || as_i64(st(1), &a.stride_b)) return nullptr;
  a.B = p;
  if (bias != Py_None) {
    int32_t kind = 0;
    int64_t dim = 2;
    if (v[21] == Py_None || v[23] == Py_None) {
      PyObject* d = PyObject_CallMethodNoArgs(bias, s_dim);
      if (!d) return nullptr;
      const int rc = as_i64(d, &dim);
      Py_DECREF(d);
      if (rc) return nullptr;
    }
    if (v[21] == Py_None) kind = dim == 1 ? XB_BIAS_ROW : XB_BIAS_FULL;
    else if (as_i32(v[21], &kind)) return nullptr;
    if (v[23] == Py_None && dim <= 1) a.ldbias = 0;
    else if (leading(v[23], bias, &a.ldbias)) return nullptr;
    if (tensor_ptr(bias, &p) || tensor_dtype(bias, &a.bias_dtype) || as_i64(st(2), &a.stride_bias) || as_i64(v[24], &a.bias_row_group))
      return nullptr;
    a.bias = p;
    a.bias_kind = kind;
  }
  if (tensor_ptr(Y, &p) || leading(v[20], Y, &a.ldy) || as_i64(st(3), &a.stride_y)) return nullptr;
  a.Y = p;
  if (as_i32(v[13], &a.batch) || tensor_dtype(A, &a.ab_dtype) || tensor_dtype(Y, &a.y_dtype) || as_i32(v[8], &a.epilogue)) return nullptr;
  const float** slots[3] = {&a.ep_a, &a.ep_b, &a.ep_c};
  for (int i = 0; i < 3; ++i) {
    PyObject* e = PyTuple_GET_ITEM(ep, i);
    if (e == Py_None) continue;
    if (tensor_ptr(e, &p)) return nullptr;
    *slots[i] = static_cast<const float*>(p);
  }
  if (as_i32(v[10], &a.ep_count) || as_flag(v[11], &a.dice_nosqrt) || as_i64(v[22], &a.stride_ep) || as_i32(v[12], &a.engine)) return nullptr;
  void* stream = PyLong_AsVoidPtr(v[25]);
  if (!stream && PyErr_Occurred()) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = api.gemm(&a, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// pool(address of the groups, how many, address and bytes of the scratch, stream) -> xb_embedding_pool's result
PyObject* py_pool(PyObject*, PyObject* const* v, Py_ssize_t n) {
  if (n != 5) { PyErr_SetString(PyExc_TypeError, "pool: 5 arguments"); return nullptr; }
  int32_t count = 0;
  int64_t bytes = 0;
  const void* groups = PyLong_AsVoidPtr(v[0]);
  void* scratch = PyLong_AsVoidPtr(v[2]);
  void* stream = PyLong_AsVoidPtr(v[4]);
  if (PyErr_Occurred() || as_i32(v[1], &count) || as_i64(v[3], &bytes)) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = api.pool(static_cast<const xb_pool_group*>(groups), count, scratch, (size_t)bytes, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// feed(predictor handle, name, C-contiguous array) -> result of ReshapeInput to the array's shape and of Feed of its bytes
PyObject* py_feed(PyObject*, PyObject* const* v, Py_ssize_t n) {
  if (n != 3) { PyErr_SetString(PyExc_TypeError, "feed: 3 arguments"); return nullptr; }
  void* handle = PyLong_AsVoidPtr(v[0]);
  if (!handle && PyErr_Occurred()) return nullptr;
  const char* name = PyUnicode_AsUTF8(v[1]);
  if (!name) return nullptr;
  Py_buffer b;
  if (PyObject_GetBuffer(v[2], &b, PyBUF_ND) != 0) return nullptr;
  std::vector<int> shape(b.ndim);
  for (int i = 0; i < b.ndim; ++i) shape[i] = (int)b.shape[i];
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = api.reshape(handle, name, shape.data(), b.ndim);
  if (rc == 0) rc = api.feed(handle, name, b.buf, (int)b.len);
  Py_END_ALLOW_THREADS
  PyBuffer_Release(&b);
  return PyLong_FromLong(rc);
}

// bind(name, address): where a C function is
PyObject* py_bind(PyObject*, PyObject* args) {
  const char* name = nullptr;
  PyObject* at = nullptr;
  if (!PyArg_ParseTuple(args, "sO", &name, &at)) return nullptr;
  void* f = PyLong_AsVoidPtr(at);
  if (!f) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
    return nullptr;
  }
  if (!strcmp(name, "xb_gemm")) api.gemm = reinterpret_cast<decltype(api.gemm)>(f);
  else if (!strcmp(name, "xb_embedding_pool")) api.pool = reinterpret_cast<decltype(api.pool)>(f);
  else if (!strcmp(name, "Blaze_PredictorReshapeInput")) api.reshape = reinterpret_cast<decltype(api.reshape)>(f);
  else if (!strcmp(name, "Blaze_PredictorFeed")) api.feed = reinterpret_cast<decltype(api.feed)>(f);
  else { PyErr_Format(PyExc_KeyError, "bind: %s", name); return nullptr; }
  Py_RETURN_NONE;
}

// dtypes({torch dtype: code})
PyObject* py_dtypes(PyObject*, PyObject* d) {
  if (!PyDict_Check(d)) { PyErr_SetString(PyExc_TypeError, "dtypes: a dict"); return nullptr; }
  Py_INCREF(d);
  Py_XSETREF(g_dtypes, d);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gemm)), METH_FASTCALL, nullptr},
    {"pool", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_pool)), METH_FASTCALL, nullptr},
    {"feed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_feed)), METH_FASTCALL, nullptr},
    {"bind", py_bind, METH_VARARGS, nullptr},
    {"dtypes", py_dtypes, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "xb_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_xb_binding(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_dtype = PyUnicode_InternFromString("dtype");
  s_stride = PyUnicode_InternFromString("stride");
  s_dim = PyUnicode_InternFromString("dim");
  g_minus2 = PyLong_FromLong(-2);
  g_dtypes = PyDict_New();
  if (!s_data_ptr || !s_dtype || !s_stride || !s_dim || !g_minus2 || !g_dtypes) return nullptr;
  return PyModule_Create(&module);
}
