/* Calls of the C ABI from Python without ctypes' per-argument conversion objects.
 *
 * A convolution takes 26 arguments; converting them through ctypes costs several microseconds, as much as the
 * kernel launch behind it, and small layers are bound by exactly that.  Every argument of the hot entry points is
 * an integer or a pointer (an int, or None for NULL), and the System V x86-64 calling convention passes each of them
 * in one 8-byte register or stack slot whatever its declared width, so one call through a function type of N
 * 64-bit integers serves them all.  The launch counter of the entry point is bumped here as well. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the argument passing below is that of x86-64 Linux"
#endif

#define MAX_ARGS 28

typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* address;
  Py_ssize_t nargs;
  PyObject* name;
  PyObject* counts; /* dict: name -> kernels launched */
  PyObject* per_call;
} FastCall;

static int to_slot(PyObject* o, int64_t* slot) {
  if (o == Py_None) {
    *slot = 0;
    return 0;
  }
  if (PyLong_Check(o)) {
    int overflow = 0;
    const long long v = PyLong_AsLongLongAndOverflow(o, &overflow);
    if (overflow > 0) {
      *slot = (int64_t)PyLong_AsUnsignedLongLong(o);
      return PyErr_Occurred() ? -1 : 0;
    }
    if (overflow < 0 || (v == -1 && PyErr_Occurred())) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_OverflowError, "argument does not fit 64 bits");
      return -1;
    }
    *slot = v;
    return 0;
  }
  PyObject* i = PyNumber_Index(o);
  if (!i) return -1;
  const int rc = to_slot(i, slot);
  Py_DECREF(i);
  return rc;
}

typedef int64_t A;
static int invoke(void* f, Py_ssize_t n, const A* a) {
  /* Registers first, then stack slots: a callee that takes fewer arguments does not look at the rest. */
  if (n <= 6) return ((int (*)(A, A, A, A, A, A))f)(a[0], a[1], a[2], a[3], a[4], a[5]);
  if (n <= 14)
    return ((int (*)(A, A, A, A, A, A, A, A, A, A, A, A, A, A))f)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9],
                                                                a[10], a[11], a[12], a[13]);
  return ((int (*)(A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A, A))f)(
      a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18],
      a[19], a[20], a[21], a[22], a[23], a[24], a[25], a[26], a[27]);
}

static PyObject* fastcall_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  FastCall* self = (FastCall*)callable;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != self->nargs || (kwnames && PyTuple_GET_SIZE(kwnames))) {
    PyErr_Format(PyExc_TypeError, "%U takes %zd positional arguments (%zd given)", self->name, self->nargs, n);
    return NULL;
  }
  A slots[MAX_ARGS] = {0};
  for (Py_ssize_t i = 0; i < n; ++i)
    if (to_slot(args[i], &slots[i])) return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS rc = invoke(self->address, n, slots);
  Py_END_ALLOW_THREADS
  if (self->per_call != Py_None) {
    PyObject* old = PyDict_GetItemWithError(self->counts, self->name); /* borrowed */
    if (!old && PyErr_Occurred()) return NULL;
    PyObject* sum = old ? PyNumber_Add(old, self->per_call) : Py_NewRef(self->per_call);
    if (!sum || PyDict_SetItem(self->counts, self->name, sum)) {
      Py_XDECREF(sum);
      return NULL;
    }
    Py_DECREF(sum);
  }
  return PyLong_FromLong(rc);
}

static void fastcall_dealloc(FastCall* self) {
  Py_XDECREF(self->name);
  Py_XDECREF(self->counts);
  Py_XDECREF(self->per_call);
  Py_TYPE(self)->tp_free((PyObject*)self);
}

static PyMemberDef fastcall_members[] = {{"__vectorcalloffset__", Py_T_PYSSIZET, offsetof(FastCall, vectorcall), Py_READONLY},
                                         {NULL}};
static PyType_Slot fastcall_slots[] = {{Py_tp_dealloc, fastcall_dealloc}, {Py_tp_call, PyVectorcall_Call},
                                       {Py_tp_members, fastcall_members}, {0, NULL}};
static PyType_Spec fastcall_spec = {"_fastcall.FastCall", sizeof(FastCall), 0,
                                    Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_DISALLOW_INSTANTIATION,
                                    fastcall_slots};
static PyTypeObject* fastcall_type;

/* bind(address, nargs, name, counts, kernels per call or None) -> callable returning the int status */
static PyObject* bind(PyObject* mod, PyObject* args) {
  unsigned long long address;
  Py_ssize_t nargs;
  PyObject *name, *counts, *per_call;
  if (!PyArg_ParseTuple(args, "KnUO!O", &address, &nargs, &name, &PyDict_Type, &counts, &per_call)) return NULL;
  if (!address || nargs < 0 || nargs > MAX_ARGS) {
    PyErr_SetString(PyExc_ValueError, "bad address or argument count");
    return NULL;
  }
  FastCall* self = PyObject_New(FastCall, fastcall_type);
  if (!self) return NULL;
  self->vectorcall = fastcall_call;
  self->address = (void*)(uintptr_t)address;
  self->nargs = nargs;
  self->name = Py_NewRef(name);
  self->counts = Py_NewRef(counts);
  self->per_call = Py_NewRef(per_call);
  return (PyObject*)self;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(address, nargs, name, counts, kernels_per_call)"}, {NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods};

PyMODINIT_FUNC PyInit__fastcall(void) {
  fastcall_type = (PyTypeObject*)PyType_FromSpec(&fastcall_spec);
  return fastcall_type ? PyModule_Create(&module) : NULL;
}
