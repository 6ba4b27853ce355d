// Calls the kernel libraries' launchers from Python: `Launcher(address, kinds, otherwise)` is a callable with one character a
// parameter ("p" pointer, "l" 64-bit, "i" 32-bit whole number, "f" float) that returns the launcher's int.
//
// ctypes takes 2.8 us to turn 26 arguments into a foreign call, a fifth of what a launch costs the host; a step of a short prompt
// launches its first kernels one after the other onto an idle GPU, so that time is the step's. Here the same call takes 0.3 us.
//
// One call form serves every signature: by the x86-64 System V calling convention whole numbers and pointers travel in their own six
// registers and then the stack, 8 bytes each, in order, and up to eight floats in theirs, whatever order the parameters are mixed in;
// the caller clears the stack, so arguments past the last parameter are ignored. A launcher with more than eight floats is refused, and
// so is any other platform; an argument that is neither a number nor None goes to `otherwise`, the ctypes function. The interpreter's lock is released
// during the call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

#define MAX_WHOLE 48
#define MAX_FLOAT 8

typedef int (*entry)(int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, float, float, float, float, float, float, float, float,
                     int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                     int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                     int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                     int64_t, int64_t, int64_t);

typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  entry fn;
  PyObject* otherwise;
  Py_ssize_t n;
  char kinds[MAX_WHOLE + MAX_FLOAT];
} Launcher;

static PyObject* launcher_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Launcher* self = (Launcher*)callable;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != self->n || (kwnames && PyTuple_GET_SIZE(kwnames))) return PyObject_Vectorcall(self->otherwise, args, nargsf, kwnames);
  int64_t w[MAX_WHOLE];
  float f[MAX_FLOAT] = {0};
  int nw = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* a = args[i];
    if (self->kinds[i] == 'f') {
      const double d = PyFloat_AsDouble(a);
      if (d == -1.0 && PyErr_Occurred()) return NULL;
      f[nf++] = (float)d;
    } else if (a == Py_None && self->kinds[i] == 'p') {
      w[nw++] = 0;
    } else if (PyLong_Check(a)) {
      const int64_t v = (int64_t)PyLong_AsUnsignedLongLongMask(a);      // (as ctypes does: the low bits, no range check)
      if (v == -1 && PyErr_Occurred()) return NULL;
      w[nw++] = v;
    } else {
      return PyObject_Vectorcall(self->otherwise, args, nargsf, kwnames);
    }
  }
  while (nw < MAX_WHOLE) w[nw++] = 0;
  int r;
  Py_BEGIN_ALLOW_THREADS
  r = self->fn(w[0], w[1], w[2], w[3], w[4], w[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], w[6], w[7], w[8], w[9], w[10], w[11],
               w[12], w[13], w[14], w[15], w[16], w[17], w[18], w[19], w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27], w[28],
               w[29], w[30], w[31], w[32], w[33], w[34], w[35], w[36], w[37], w[38], w[39], w[40], w[41], w[42], w[43], w[44], w[45],
               w[46], w[47]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(r);
}

static PyObject* launcher_new(PyTypeObject* type, PyObject* args, PyObject* kwargs) {
  unsigned long long address;
  const char* kinds;
  Py_ssize_t n;
  PyObject* otherwise;
  if (!PyArg_ParseTuple(args, "Ks#O", &address, &kinds, &n, &otherwise)) return NULL;
  int nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (kinds[i] == 'f') ++nf;
    else if (kinds[i] != 'p' && kinds[i] != 'l' && kinds[i] != 'i') {
      PyErr_Format(PyExc_ValueError, "parameter kind %c", kinds[i]);
      return NULL;
    }
  }
  if (nf > MAX_FLOAT || n - nf > MAX_WHOLE) {
    PyErr_SetString(PyExc_ValueError, "too many parameters");
    return NULL;
  }
  Launcher* self = (Launcher*)type->tp_alloc(type, 0);
  if (!self) return NULL;
  self->vectorcall = launcher_call;
  self->fn = (entry)(uintptr_t)address;
  self->otherwise = Py_NewRef(otherwise);
  self->n = n;
  for (Py_ssize_t i = 0; i < n; ++i) self->kinds[i] = kinds[i];
  return (PyObject*)self;
}

static void launcher_dealloc(PyObject* o) {
  Py_XDECREF(((Launcher*)o)->otherwise);
  Py_TYPE(o)->tp_free(o);
}

// What is not the launcher's own is the ctypes function's (argtypes, restype).
static PyObject* launcher_getattr(PyObject* o, PyObject* name) {
  PyObject* own = PyObject_GenericGetAttr(o, name);
  if (own || !PyErr_ExceptionMatches(PyExc_AttributeError)) return own;
  PyErr_Clear();
  return PyObject_GetAttr(((Launcher*)o)->otherwise, name);
}

static PyTypeObject launcher_type = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "fastcall.Launcher",
    .tp_basicsize = sizeof(Launcher),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_new = launcher_new,
    .tp_dealloc = launcher_dealloc,
    .tp_call = PyVectorcall_Call,
    .tp_getattro = launcher_getattr,
    .tp_vectorcall_offset = offsetof(Launcher, vectorcall),
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "fastcall", NULL, -1, NULL};

PyMODINIT_FUNC PyInit_fastcall(void) {
#if !defined(__x86_64__) || defined(_WIN32)
  PyErr_SetString(PyExc_ImportError, "written for x86-64 System V");
  return NULL;
#endif
  if (PyType_Ready(&launcher_type) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddObjectRef(m, "Launcher", (PyObject*)&launcher_type) < 0) Py_CLEAR(m);
  return m;
}
