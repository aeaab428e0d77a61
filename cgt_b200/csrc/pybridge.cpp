// CPython module `cgt_b200._pybridge`: the call of a compiled function without ctypes.
//
// run(interp, types, args, wrapper_type) takes the arguments of one call (numpy arrays of exactly the declared dtype and
// rank in C order, or ArrayWrapper objects), runs the interpreter without the GIL and returns the outputs as new numpy
// arrays. It returns NotImplemented, having done nothing, when an argument needs a conversion: runtime.py then takes the
// general path. What it saves is host time between calls: a ctypes call costs about half a microsecond, the general path
// makes a dozen of them for one argument and one result.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstring>
#include "../../include/cgt_b200.h"

namespace {

PyObject *g_empty = nullptr, *g_ndarray = nullptr, *g_handle_name = nullptr;
PyObject* g_dtypes[32] = {nullptr};  // by numpy type number

bool format_is(const Py_buffer& v, int type_num) {
  const char* f = v.format ? v.format : "B";
  if (*f == '@' || *f == '=' || *f == '<') ++f;
  if (f[0] == 0 || f[1] != 0) return false;
  switch (type_num) {
    case cgtb_i1: return f[0] == 'b';
    case cgtb_i2: return f[0] == 'h';
    case cgtb_i4: return f[0] == 'i' || (f[0] == 'l' && v.itemsize == 4);
    case cgtb_i8: return (f[0] == 'l' || f[0] == 'q') && v.itemsize == 8;
    case cgtb_f4: return f[0] == 'f';
    case cgtb_f8: return f[0] == 'd';
  }
  return false;
}

PyObject* to_numpy(cgtbInterp* it, int i, cgtbObject* o) {
  if (cgtb_object_kind(o) != 1) return nullptr;  // runtime.py keeps functions with tuple results away
  const int nd = cgtb_array_ndim(o), dt = cgtb_array_dtype(o);
  if (dt < 0 || dt >= 32 || !g_dtypes[dt]) return nullptr;
  const long* shp = cgtb_array_shape(o);
  PyObject* shape = PyTuple_New(nd);
  if (!shape) return nullptr;
  for (int d = 0; d < nd; ++d) PyTuple_SET_ITEM(shape, d, PyLong_FromLong(shp[d]));
  PyObject* out = PyObject_CallFunctionObjArgs(g_empty, shape, g_dtypes[dt], nullptr);
  Py_DECREF(shape);
  if (!out) return nullptr;
  Py_buffer v;
  if (PyObject_GetBuffer(out, &v, PyBUF_WRITABLE) != 0) { Py_DECREF(out); return nullptr; }
  const long n = cgtb_array_nbytes(o);
  int rc = 0;
  if (n > 0) {
    const void* host = cgtb_interp_output_host(it, i);
    if (!host && cgtb_array_devtype(o) == cgtbCPU) host = cgtb_array_data(o);
    if (host) cgtb_host_copy(v.buf, host, n);
    else rc = cgtb_array_to_host(o, v.buf);
  }
  PyBuffer_Release(&v);
  if (rc) {
    Py_DECREF(out);
    PyErr_SetString(PyExc_RuntimeError, cgtb_last_error());
    return nullptr;
  }
  return out;
}

// run(interp: int, types: bytes of (type number, rank) pairs, args: tuple, wrapper_type) -> list or NotImplemented
PyObject* run(PyObject*, PyObject* const* a, Py_ssize_t na) {
  if (na != 4 || !PyBytes_Check(a[1]) || !PyTuple_Check(a[2]) || !PyType_Check(a[3])) {
    PyErr_SetString(PyExc_TypeError, "run(interp, types, args, wrapper_type)");
    return nullptr;
  }
  cgtbInterp* it = (cgtbInterp*)PyLong_AsVoidPtr(a[0]);
  if (!it) return PyErr_Occurred() ? nullptr : (PyErr_SetString(PyExc_ValueError, "null interpreter"), nullptr);
  PyObject* args = a[2];
  const Py_ssize_t n = PyTuple_GET_SIZE(args);
  constexpr Py_ssize_t kMax = 32;
  if (n > kMax || PyBytes_GET_SIZE(a[1]) != 2 * n) Py_RETURN_NOTIMPLEMENTED;
  const unsigned char* types = (const unsigned char*)PyBytes_AS_STRING(a[1]);
  Py_buffer views[kMax];
  bool held[kMax];
  cgtbObject* objs[kMax];
  bool usable = true;
  Py_ssize_t k = 0;
  for (; k < n && usable; ++k) {
    PyObject* o = PyTuple_GET_ITEM(args, k);
    held[k] = false;
    objs[k] = nullptr;
    if (Py_TYPE(o) == (PyTypeObject*)a[3]) {
      PyObject* h = PyObject_GetAttr(o, g_handle_name);
      if (h && PyLong_Check(h)) {
        objs[k] = (cgtbObject*)PyLong_AsVoidPtr(h);
        if (objs[k]) cgtb_retain(objs[k]);
      }
      Py_XDECREF(h);
      usable = objs[k] != nullptr;
    } else if ((PyObject*)Py_TYPE(o) == g_ndarray) {
      if (PyObject_GetBuffer(o, &views[k], PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) {
        usable = false;
        break;
      }
      held[k] = true;
      const Py_buffer& v = views[k];
      if (!format_is(v, types[2 * k]) || v.ndim != types[2 * k + 1] || v.ndim > 8) usable = false;
      else {
        long shape[8] = {0};
        for (int d = 0; d < v.ndim; ++d) shape[d] = (long)v.shape[d];
        objs[k] = cgtb_array_from_host(v.ndim, shape, types[2 * k], cgtbCPU, v.buf, 0);
        usable = objs[k] != nullptr;
      }
    } else {
      usable = false;
    }
  }
  const Py_ssize_t made = k;
  PyErr_Clear();
  cgtbObject* out = nullptr;
  int rc = 0;
  if (usable) {
    cgtbObject* cargs = cgtb_tuple_new((int)n);
    for (Py_ssize_t i = 0; i < n; ++i) cgtb_tuple_set(cargs, (int)i, objs[i]);
    Py_BEGIN_ALLOW_THREADS
    rc = cgtb_interp_run(it, cargs, &out);
    Py_END_ALLOW_THREADS
    cgtb_release(cargs);
  }
  for (Py_ssize_t i = 0; i < made; ++i) {
    if (objs[i]) cgtb_release(objs[i]);
    if (held[i]) PyBuffer_Release(&views[i]);
  }
  if (!usable) Py_RETURN_NOTIMPLEMENTED;
  if (rc) return PyLong_FromLong(rc);  // the caller reports it
  const int n_out = cgtb_tuple_len(out);
  PyObject* res = PyList_New(n_out);
  for (int i = 0; res && i < n_out; ++i) {
    PyObject* v = to_numpy(it, i, cgtb_tuple_get(out, i));
    if (!v) { Py_CLEAR(res); break; }
    PyList_SET_ITEM(res, i, v);
  }
  if (!res) {
    cgtb_release(out);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "an output has an unknown type");
    return nullptr;
  }
  cgtb_release(out);
  return res;
}

PyMethodDef methods[] = {{"run", (PyCFunction)(void (*)(void))run, METH_FASTCALL, "One call of a compiled function."}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pybridge", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pybridge(void) {
  PyObject* np = PyImport_ImportModule("numpy");
  if (!np) return nullptr;
  g_empty = PyObject_GetAttrString(np, "empty");
  g_ndarray = PyObject_GetAttrString(np, "ndarray");
  g_handle_name = PyUnicode_InternFromString("handle");
  const struct { int num; const char* name; } dts[] = {{cgtb_i1, "int8"}, {cgtb_i2, "int16"}, {cgtb_i4, "int32"}, {cgtb_i8, "int64"},
                                                       {cgtb_f4, "float32"}, {cgtb_f8, "float64"}};
  for (auto& d : dts) {
    PyObject* name = PyUnicode_FromString(d.name);
    PyObject* f = PyObject_GetAttrString(np, "dtype");
    g_dtypes[d.num] = f && name ? PyObject_CallOneArg(f, name) : nullptr;
    Py_XDECREF(name);
    Py_XDECREF(f);
    if (!g_dtypes[d.num]) return nullptr;
  }
  Py_DECREF(np);
  if (!g_empty || !g_ndarray || !g_handle_name) return nullptr;
  return PyModule_Create(&module);
}
