// Calls the library's launchers from Python without ctypes: one C call per launch, arguments read in place.
//
// A launcher takes integers, pointers and at most eight single-precision floats, in any order.  The System V x86-64 calling
// convention hands the first six integers over in general registers, floats in vector registers, and the remaining integers on
// the stack in their order, each kind counted by itself.  So one prototype -- integers and floats apart, more stack slots than
// any launcher reads -- calls them all; a 32-bit parameter reads the low half of its slot.  A call of 14 arguments takes 0.7 us
// of host time before the launch itself, 4.0 us through ctypes; a training step of two small layers makes 61 of them.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the argument passing below is that of x86-64 System V"
#endif

enum { MAX_INTS = 48, MAX_FLOATS = 8 };

typedef int (*Fn)(long, long, long, long, long, long, float, float, float, float, float, float, float, float, long, long, long,
                  long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                  long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long,
                  long, long, long);

typedef struct {
  PyObject_HEAD
  vectorcallfunc call;
  Fn fn;
  Py_ssize_t n;                        // arguments, without the stream
  int stream;                          // the call appends one
  char kinds[MAX_INTS + MAX_FLOATS];   // 'f' float, 'l' integer, 'p' pointer
} Launcher;

static PyObject *tensor_type, *data_ptr_name;

// one argument of kind 'l' or 'p'; 0: not one of that kind
static int as_integer(PyObject* a, char kind, long* out) {
  if (PyLong_Check(a)) {
    *out = (long)PyLong_AsUnsignedLongLongMask(a);
  } else if (a == Py_None && kind == 'p') {
    *out = 0;
  } else if (PyObject_TypeCheck(a, (PyTypeObject*)tensor_type)) {
    PyObject* p = PyObject_CallMethodNoArgs(a, data_ptr_name);
    if (!p) return 0;
    *out = (long)PyLong_AsUnsignedLongLongMask(p);
    Py_DECREF(p);
  } else if (kind == 'p' && PyBytes_Check(a)) {
    *out = (long)PyBytes_AS_STRING(a);
  } else {
    return 0;
  }
  return !(*out == -1 && PyErr_Occurred());
}

// launcher(args, stream) -> return code; None: an argument is of another kind than the launcher was bound with
static PyObject* launcher_call(PyObject* self, PyObject* const* argv, size_t nargsf, PyObject* kwnames) {
  Launcher* l = (Launcher*)self;
  if (PyVectorcall_NARGS(nargsf) != 2 || kwnames || !PyTuple_Check(argv[0]) || !PyLong_Check(argv[1])) {
    PyErr_SetString(PyExc_TypeError, "launcher(args, stream)");
    return NULL;
  }
  PyObject* args = argv[0];
  if (PyTuple_GET_SIZE(args) != l->n) Py_RETURN_NONE;
  long v[MAX_INTS] = {0};
  float f[MAX_FLOATS] = {0};
  int nv = 0, nf = 0;
  for (Py_ssize_t i = 0; i < l->n; ++i) {
    PyObject* a = PyTuple_GET_ITEM(args, i);
    if (l->kinds[i] == 'f') {
      if (!PyFloat_Check(a) && !PyLong_Check(a)) Py_RETURN_NONE;
      const double d = PyFloat_AsDouble(a);
      if (d == -1. && PyErr_Occurred()) return NULL;
      f[nf++] = (float)d;
    } else if (!as_integer(a, l->kinds[i], &v[nv++])) {
      if (PyErr_Occurred()) return NULL;
      Py_RETURN_NONE;
    }
  }
  if (l->stream) v[nv++] = (long)PyLong_AsUnsignedLongLongMask(argv[1]);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = l->fn(v[0], v[1], v[2], v[3], v[4], v[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], v[6], v[7], v[8], v[9], v[10],
             v[11], v[12], v[13], v[14], v[15], v[16], v[17], v[18], v[19], v[20], v[21], v[22], v[23], v[24], v[25], v[26],
             v[27], v[28], v[29], v[30], v[31], v[32], v[33], v[34], v[35], v[36], v[37], v[38], v[39], v[40], v[41], v[42],
             v[43], v[44], v[45], v[46], v[47]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyTypeObject LauncherType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "primus_b200._launch.Launcher",
    .tp_basicsize = sizeof(Launcher),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Launcher, call),
    .tp_call = PyVectorcall_Call,
};

// bind(address, kinds, stream) -> launcher, or None if there are more arguments than the prototype has room for
static PyObject* bind(PyObject* self, PyObject* args) {
  unsigned long long address;
  const char* kinds;
  Py_ssize_t n;
  int stream;
  if (!PyArg_ParseTuple(args, "Ky#p", &address, &kinds, &n, &stream)) return NULL;
  Py_ssize_t floats = 0;
  for (Py_ssize_t i = 0; i < n; ++i) floats += kinds[i] == 'f';
  if (floats > MAX_FLOATS || n - floats + stream > MAX_INTS) Py_RETURN_NONE;
  Launcher* l = PyObject_New(Launcher, &LauncherType);
  if (!l) return NULL;
  l->call = launcher_call;
  l->fn = (Fn)address;
  l->n = n;
  l->stream = stream;
  memcpy(l->kinds, kinds, n);
  return (PyObject*)l;
}

// init(tensor type): what counts as a tensor
static PyObject* init(PyObject* self, PyObject* type) {
  if (!PyType_Check(type)) {
    PyErr_SetString(PyExc_TypeError, "a type");
    return NULL;
  }
  Py_XDECREF(tensor_type);
  tensor_type = Py_NewRef(type);
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, NULL}, {"init", init, METH_O, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launch", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__launch(void) {
  if (PyType_Ready(&LauncherType) < 0) return NULL;
  data_ptr_name = PyUnicode_InternFromString("data_ptr");
  return data_ptr_name ? PyModule_Create(&module) : NULL;
}
