// Calls of the quantized linears' C functions from Python without ctypes: an argument block built from keyword fields and a foreign call cost some
// 3 us, a quarter of what a one-row linear takes from call to call; a vectorcall function with plain integers costs 0.3.  The functions' addresses come
// from the library as it is loaded (bind); nothing else is kept.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>

#include "../../include/b2l.h"

namespace {

using Q4Fn = int (*)(const b2l_q4_linear_args*, b2l_stream_t);
using Q8Fn = int (*)(const void*, int, const void*, const void*, void*, int, void*, int, int, int, float, b2l_stream_t);
Q4Fn q4_fn[4];
Q8Fn q8_fn;

void* ptr(PyObject* o) { return o == Py_None ? nullptr : PyLong_AsVoidPtr(o); }
int num(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v != (long)(int)v && !PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "size outside 32 bits");
  return (int)v;
}
bool takes(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) PyErr_Format(PyExc_TypeError, "%zd arguments, %zd wanted", got, want);
  return got == want;
}

// bind(q4_gemv, q4_gemv_batch, q4_linear_tc, q4_gemm, q8_linear): addresses
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!takes(n, 5)) return nullptr;
  for (int i = 0; i < 4; ++i) q4_fn[i] = reinterpret_cast<Q4Fn>(ptr(a[i]));
  q8_fn = reinterpret_cast<Q8Fn>(ptr(a[4]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// q4(which, x, ldx, qw_tiled, scales, zeros, sz_dtype, y, ldy, M, N, K, workspace, stream) -> return code
PyObject* q4(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!takes(n, 14)) return nullptr;
  const int which = num(a[0]);
  b2l_q4_linear_args q = {};
  q.x = ptr(a[1]); q.ldx = num(a[2]);
  q.qw_tiled = ptr(a[3]); q.scales = ptr(a[4]); q.zeros = ptr(a[5]); q.sz_dtype = num(a[6]);
  q.y = ptr(a[7]); q.ldy = num(a[8]);
  q.M = num(a[9]); q.N = num(a[10]); q.K = num(a[11]);
  q.workspace = ptr(a[12]);
  void* stream = ptr(a[13]);
  if (PyErr_Occurred()) return nullptr;
  if (which < 0 || which > 3 || !q4_fn[which]) return PyErr_Format(PyExc_RuntimeError, "function %d is not bound", which);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = q4_fn[which](&q, (b2l_stream_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// q8(x, ldx, cb, scb, y, ldy, workspace, M, N, K, threshold, stream) -> return code
PyObject* q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!takes(n, 12)) return nullptr;
  void *x = ptr(a[0]), *cb = ptr(a[2]), *scb = ptr(a[3]), *y = ptr(a[4]), *ws = ptr(a[6]), *stream = ptr(a[11]);
  const int ldx = num(a[1]), ldy = num(a[5]), M = num(a[7]), N = num(a[8]), K = num(a[9]);
  const double threshold = PyFloat_AsDouble(a[10]);
  if (PyErr_Occurred()) return nullptr;
  if (!q8_fn) return PyErr_Format(PyExc_RuntimeError, "q8 is not bound");
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = q8_fn(x, ldx, cb, scb, y, ldy, ws, M, N, K, (float)threshold, (b2l_stream_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

PyMethodDef methods[] = {{"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
                         {"q4", (PyCFunction)(void (*)(void))q4, METH_FASTCALL, nullptr},
                         {"q8", (PyCFunction)(void (*)(void))q8, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall(void) { return PyModule_Create(&module_def); }
