// Python calls of the library's launchers without ctypes.
//
// A step of small kernels is bound by the host, and ctypes took 2.3 us of a call of 16 arguments, half of what the launch itself
// takes.  Here it is 0.7 us (0.6B width, 3 rows of 333, a training step of 170
// calls: 6.38 -> 6.08 ms): the arguments arrive as an array, are converted by a function made for the launcher's signature and the
// GIL is released around the call, as ctypes does.  table.inc, written by the build, has one line SIG(name, types...) per launcher of
// lib.py; addresses come from the library that lib.py has loaded.  What the table does not cover (other launchers,
// arguments that are no numbers) is left to ctypes: call() returns None.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>
#include <tuple>
#include <utility>

namespace {

using P = void*;
using I = int;
using L = long long;
using U = unsigned;
using F = float;
using D = double;

bool get(PyObject* o, P& v) {
  if (o == Py_None) v = nullptr;
  else if (PyLong_Check(o)) v = reinterpret_cast<P>(PyLong_AsUnsignedLongLongMask(o));
  else return false;
  return true;
}
template <typename T>
bool get_int(PyObject* o, T& v) {
  if (!PyLong_Check(o)) return false;
  v = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
  return true;
}
bool get(PyObject* o, I& v) { return get_int(o, v); }
bool get(PyObject* o, L& v) { return get_int(o, v); }
bool get(PyObject* o, U& v) { return get_int(o, v); }
bool get(PyObject* o, D& v) {
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
  v = PyFloat_AsDouble(o);
  return !PyErr_Occurred();
}
bool get(PyObject* o, F& v) {
  D d;
  if (!get(o, d)) return false;
  v = static_cast<F>(d);
  return true;
}

template <typename... A>
struct Launcher {
  static constexpr int kArgs = sizeof...(A);
  template <size_t... K>
  static bool convert(PyObject* const* a, std::tuple<A...>& t, std::index_sequence<K...>) {
    return (get(a[K], std::get<K>(t)) && ...);
  }
  static bool run(void* f, PyObject* const* a, int* rc) {
    std::tuple<A...> t;
    if (!convert(a, t, std::index_sequence_for<A...>())) return false;
    Py_BEGIN_ALLOW_THREADS
    *rc = std::apply(reinterpret_cast<int (*)(A...)>(f), t);
    Py_END_ALLOW_THREADS
    return true;
  }
};

struct Entry {
  const char* name;
  int args;
  bool (*run)(void*, PyObject* const*, int*);
  void* address;
};
#define SIG(name, ...) {#name, Launcher<__VA_ARGS__>::kArgs, Launcher<__VA_ARGS__>::run, nullptr},
Entry entries[] = {
#include "table.inc"
};
PyObject* by_name;      // name -> index, int

PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyUnicode_Check(a[0]) || !PyLong_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "bind(name, address)");
    return nullptr;
  }
  PyObject* at = PyDict_GetItemWithError(by_name, a[0]);
  if (at) entries[PyLong_AsLong(at)].address = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(a[1]));
  else if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyObject* call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n < 1) Py_RETURN_NONE;
  PyObject* at = PyDict_GetItemWithError(by_name, a[0]);
  if (!at) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const Entry& e = entries[PyLong_AsLong(at)];
  int rc = 0;
  if (!e.address || e.args != n - 1 || !e.run(e.address, a + 1, &rc)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  return PyLong_FromLong(rc);
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, "bind(name, address): 0 takes it back"},
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call)), METH_FASTCALL, "call(name, ...) -> code, or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch() {
  PyObject* m = PyModule_Create(&module);
  by_name = PyDict_New();
  if (!m || !by_name) return nullptr;
  const int n = sizeof(entries) / sizeof(entries[0]);
  for (int i = 0; i < n; ++i) {
    PyObject* v = PyLong_FromLong(i);
    if (!v || PyDict_SetItemString(by_name, entries[i].name, v)) return nullptr;
    Py_DECREF(v);
  }
  if (PyModule_AddStringConstant(m, "signatures", SIGNATURES)) return nullptr;
  return m;
}
