// Calls of the sequence kernels' C functions from Python without ctypes.  A portion is many small launches (eager, 64 for four layers) whose host side bounds it up
// to some hundred tokens, and ctypes converts an argument in 0.25 us: 5.7 us for a rotation's 20 arguments, 3.3 for a norm's 11 (the functions return at once
// for no tokens, so that is the call alone).  A function made here takes 0.3 and 0.25: the delta layer's pass of up to some hundred tokens lost 12 of 120 us,
// latent attention's 10 of 112, the host side of a replayed four-layer portion went from 115 to 75.  What converts without loss (integers in range, floats,
// None for a pointer) is converted here; every other call goes, with its errors, to the ctypes function that it stands for.  The types come from the
// declarations, and the caller's signature string must equal theirs, or nothing is made.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>
#include <cstdint>
#include <cstring>
#include <new>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/b2l_seq.h"

namespace {

template <class T> constexpr char code() {
  static_assert(std::is_pointer_v<T> || std::is_same_v<T, float> || std::is_same_v<T, int> || std::is_same_v<T, long long> || std::is_same_v<T, size_t>);
  return std::is_pointer_v<T> ? 'p' : std::is_same_v<T, float> ? 'f' : std::is_same_v<T, int> ? 'i' : std::is_same_v<T, long long> ? 'q' : 'z';
}

// the argument as T; `fits` becomes false (an exception may be set) where ctypes has to decide
template <class T> T get(PyObject* o, bool& fits) {
  if constexpr (std::is_same_v<T, float>) {
    if (PyFloat_Check(o)) return (float)PyFloat_AsDouble(o);
    fits = false;
    return 0.f;
  } else if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    if (!PyLong_Check(o)) return fits = false, nullptr;
    const unsigned long long v = PyLong_AsUnsignedLongLong(o);
    if (v == ~0ull) fits = false;                        // too large, negative, or that address
    return reinterpret_cast<T>((uintptr_t)v);
  } else {
    if (!PyLong_Check(o)) return fits = false, T(0);
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) fits = false;
    if (std::is_same_v<T, int> ? v < INT_MIN || v > INT_MAX : std::is_same_v<T, size_t> && v < 0) fits = false;
    return (T)v;
  }
}

template <class F> struct Thunk;
template <class... A> struct Thunk<int (*)(A...)> {
  static constexpr char signature[] = {code<A>()..., 0};
  template <size_t... I> static bool go(void* fn, PyObject* const* a, int* rc, std::index_sequence<I...>) {
    bool fits = true;
    const std::tuple<A...> v{get<A>(a[I], fits)...};
    if (!fits) return false;
    Py_BEGIN_ALLOW_THREADS
    *rc = reinterpret_cast<int (*)(A...)>(fn)(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return true;
  }
  static bool call(void* fn, PyObject* const* a, int* rc) { return go(fn, a, rc, std::make_index_sequence<sizeof...(A)>()); }
};

struct Entry {
  const char *name, *signature;
  bool (*call)(void*, PyObject* const*, int*);
};
#define ALL(F) \
  F(b2l_seq_embed) \
  F(b2l_seq_rmsnorm) \
  F(b2l_seq_norm_add_norm) \
  F(b2l_seq_gated_act) \
  F(b2l_seq_linear_f32) \
  F(b2l_seq_conv_silu) \
  F(b2l_seq_conv_silu_unit) \
  F(b2l_seq_unit_norm) \
  F(b2l_seq_decay) \
  F(b2l_seq_group_norm_gate) \
  F(b2l_seq_headnorm_rope) \
  F(b2l_seq_cast_f32) \
  F(b2l_seq_zero_slot) \
  F(b2l_seq_add_norm2) \
  F(b2l_seq_softcap) \
  F(b2l_seq_rope) \
  F(b2l_seq_latent_prep) \
  F(b2l_seq_moe_route) \
  F(b2l_seq_moe_route_fused) \
  F(b2l_seq_moe_experts_small) \
  F(b2l_seq_moe_sort) \
  F(b2l_seq_moe_gather) \
  F(b2l_seq_moe_combine) \
  F(b2l_seq_embed_pair) \
  F(b2l_seq_hc_step) \
  F(b2l_seq_hc_sum) \
  F(b2l_seq_scale) \
  F(b2l_seq_unary_act) \
  F(b2l_seq_diff_combine) \
  F(b2l_seq_mingru) \
  F(b2l_seq_norm) \
  F(b2l_seq_depth_step) \
  F(b2l_seq_latent_up) \
  F(b2l_seq_head_gate) \
  F(b2l_seq_linear_few)
#define ENTRY(name) {#name, Thunk<decltype(&name)>::signature, Thunk<decltype(&name)>::call},
const Entry entries[] = {ALL(ENTRY)};
constexpr int N_ENTRIES = (int)(sizeof(entries) / sizeof(entries[0]));

struct Bound {
  const Entry* e;
  void* fn;
  PyObject* slow;                                        // the ctypes function: this one's owner while it lives, and the library's
  Py_ssize_t n;
};
constexpr char CAPSULE[] = "b2l_seq function";

PyObject* invoke(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  const Bound* b = (const Bound*)PyCapsule_GetPointer(self, CAPSULE);
  if (!b) return nullptr;
  int rc;
  if (n == b->n && b->e->call(b->fn, a, &rc)) return PyLong_FromLong(rc);
  PyErr_Clear();
  PyObject* args = PyTuple_New(n);
  if (!args) return nullptr;
  for (Py_ssize_t i = 0; i < n; ++i) {
    Py_INCREF(a[i]);
    PyTuple_SetItem(args, i, a[i]);
  }
  PyObject* r = PyObject_CallObject(b->slow, args);
  Py_DECREF(args);
  return r;
}

void drop(PyObject* capsule) {
  Bound* b = (Bound*)PyCapsule_GetPointer(capsule, CAPSULE);
  if (!b) return;
  Py_XDECREF(b->slow);
  delete b;
}

#define METHOD(name) {#name, (PyCFunction)(void (*)(void))invoke, METH_FASTCALL, nullptr},
PyMethodDef functions[] = {ALL(METHOD)};

// make(name, address, ctypes function, signature) -> function, or None where this file has none of that name and signature
PyObject* make(PyObject*, PyObject* args) {
  const char *name, *signature;
  PyObject *at, *slow;
  if (!PyArg_ParseTuple(args, "sOOs", &name, &at, &slow, &signature)) return nullptr;
  void* fn = PyLong_AsVoidPtr(at);
  if (PyErr_Occurred()) return nullptr;
  int i = 0;
  while (i < N_ENTRIES && std::strcmp(entries[i].name, name)) ++i;
  if (i == N_ENTRIES || !fn || std::strcmp(entries[i].signature, signature)) Py_RETURN_NONE;
  Bound* b = new (std::nothrow) Bound{&entries[i], fn, slow, (Py_ssize_t)std::strlen(signature)};
  if (!b) return PyErr_NoMemory();
  PyObject* capsule = PyCapsule_New(b, CAPSULE, drop);
  if (!capsule) {
    delete b;
    return nullptr;
  }
  Py_INCREF(slow);
  PyObject* f = PyCFunction_NewEx(&functions[i], capsule, nullptr);
  Py_DECREF(capsule);
  return f;
}

PyMethodDef methods[] = {{"make", (PyCFunction)make, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_seqcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__seqcall(void) { return PyModule_Create(&module_def); }
