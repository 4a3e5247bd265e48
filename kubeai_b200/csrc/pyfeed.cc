// kubeai_b200._feed: the entries of a fed step (Engine.feed_step) from a list of (id, tokens, wanted offsets) to the C call's
// array in one pass.  For lists of exact tuples with int ids and contiguous int32 vectors, which is what a serving loop has in
// hand; for anything else pack() answers None and the caller forms the entries with numpy, which takes 0.8 us a sequence
// (two joins, their lengths, the ids) where this takes 0.05: 101 us of a step of 128 sequences, 17 of one.
#define PY_SSIZE_T_CLEAN
#define NPY_NO_DEPRECATED_API NPY_1_7_API_VERSION
#include <Python.h>
#include <limits.h>
#include <numpy/arrayobject.h>
#include <string.h>

#include "b200engine.h"

namespace {

bool int32_vector(PyObject* o) {
  if (!PyArray_CheckExact(o)) return false;
  PyArrayObject* a = reinterpret_cast<PyArrayObject*>(o);
  return PyArray_TYPE(a) == NPY_INT32 && PyArray_NDIM(a) == 1 && PyArray_IS_C_CONTIGUOUS(a) && PyArray_ISNOTSWAPPED(a) && PyArray_DIM(a, 0) <= INT_MAX;
}

// pack(entries) -> (bytearray of b200_feed_entry and behind them the numbers they point at, wanted rows), or None.  The numbers
// are copied: the call they go to runs without the interpreter's lock.
PyObject* pack(PyObject*, PyObject* entries) {
  if (!PyList_CheckExact(entries)) Py_RETURN_NONE;
  const Py_ssize_t n = PyList_GET_SIZE(entries);
  Py_ssize_t numbers = 0, wanted = 0;
  if (n < 1 || n > INT_MAX) Py_RETURN_NONE;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* e = PyList_GET_ITEM(entries, i);
    if (!PyTuple_CheckExact(e) || PyTuple_GET_SIZE(e) != 3 || !PyLong_CheckExact(PyTuple_GET_ITEM(e, 0))) Py_RETURN_NONE;
    if (!int32_vector(PyTuple_GET_ITEM(e, 1)) || !int32_vector(PyTuple_GET_ITEM(e, 2))) Py_RETURN_NONE;
    const Py_ssize_t w = PyArray_DIM(reinterpret_cast<PyArrayObject*>(PyTuple_GET_ITEM(e, 2)), 0);
    numbers += PyArray_DIM(reinterpret_cast<PyArrayObject*>(PyTuple_GET_ITEM(e, 1)), 0) + w;
    wanted += w;
  }
  PyObject* buf = PyByteArray_FromStringAndSize(nullptr, n * static_cast<Py_ssize_t>(sizeof(b200_feed_entry)) + numbers * 4);
  if (!buf) return nullptr;
  b200_feed_entry* out = reinterpret_cast<b200_feed_entry*>(PyByteArray_AS_STRING(buf));
  int32_t* at = reinterpret_cast<int32_t*>(out + n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* e = PyList_GET_ITEM(entries, i);
    memset(&out[i], 0, sizeof(out[i]));
    out[i].req_id = PyLong_AsUnsignedLongLongMask(PyTuple_GET_ITEM(e, 0));
    auto copy = [&](PyObject* o, int32_t* count) {
      PyArrayObject* a = reinterpret_cast<PyArrayObject*>(o);
      const int32_t* from = at;
      *count = static_cast<int32_t>(PyArray_DIM(a, 0));
      if (*count) memcpy(at, PyArray_DATA(a), static_cast<size_t>(*count) * 4);
      at += *count;
      return from;
    };
    out[i].tokens = copy(PyTuple_GET_ITEM(e, 1), &out[i].n_tokens);
    out[i].want = copy(PyTuple_GET_ITEM(e, 2), &out[i].n_want);
    if (!out[i].n_want) out[i].want = nullptr;
  }
  return Py_BuildValue("Nn", buf, wanted);
}

PyMethodDef methods[] = {{"pack", pack, METH_O, "entries of a fed step as the C call takes them"}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_feed", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__feed(void) {
  import_array();
  return PyModule_Create(&module);
}
