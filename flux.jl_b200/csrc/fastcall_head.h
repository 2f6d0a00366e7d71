// Head of the generated `_fastcall` extension module: argument conversion of the wrappers and the module's own functions.
// A getter answers 0 for an object it does not take; the wrapper then returns None and the caller goes through ctypes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

static inline int get_p(PyObject* o, void** out) {
  if (o == Py_None) { *out = NULL; return 1; }
  if (!PyLong_Check(o)) return 0;
  *out = PyLong_AsVoidPtr(o);
  if (*out == NULL && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return 1;
}
static inline int get_l(PyObject* o, int64_t* out) {
  if (!PyLong_Check(o)) return 0;
  *out = PyLong_AsLongLong(o);
  if (*out == -1 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return 1;
}
static inline int get_i(PyObject* o, int32_t* out) {
  int64_t v;
  if (!get_l(o, &v) || v < INT32_MIN || v > INT32_MAX) return 0;
  *out = (int32_t)v;
  return 1;
}
static inline int get_u(PyObject* o, uint64_t* out) {
  if (!PyLong_Check(o)) return 0;
  *out = PyLong_AsUnsignedLongLong(o);
  if (*out == (uint64_t)-1 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return 1;
}
static inline int get_f(PyObject* o, float* out) {
  if (PyFloat_Check(o)) { *out = (float)PyFloat_AS_DOUBLE(o); return 1; }
  if (!PyLong_Check(o)) return 0;
  const double d = PyLong_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  *out = (float)d;
  return 1;
}

#define FASTCALL_BIND_AND_NAMES                                                                  \
  static PyObject* do_bind(PyObject* self, PyObject* args) {                                     \
    const char* name;                                                                            \
    unsigned long long addr;                                                                     \
    (void)self;                                                                                  \
    if (!PyArg_ParseTuple(args, "sK", &name, &addr)) return NULL;                                \
    for (int i = 0; slots[i].name != NULL; ++i)                                                  \
      if (strcmp(slots[i].name, name) == 0) { *slots[i].slot = (void*)(uintptr_t)addr; Py_RETURN_TRUE; } \
    Py_RETURN_FALSE;                                                                             \
  }                                                                                              \
  static PyObject* do_names(PyObject* self, PyObject* unused) {                                  \
    (void)self; (void)unused;                                                                    \
    PyObject* l = PyList_New(0);                                                                 \
    for (int i = 0; l != NULL && slots[i].name != NULL; ++i) {                                   \
      PyObject* u = PyUnicode_FromString(slots[i].name);                                         \
      if (u == NULL || PyList_Append(l, u) != 0) { Py_XDECREF(u); Py_CLEAR(l); break; }          \
      Py_DECREF(u);                                                                              \
    }                                                                                            \
    return l;                                                                                    \
  }

#define FASTCALL_MODULE                                                                                        \
  static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL}; \
  PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
