/* Launchers of libatb.so as Python callables with declared argument types ("ppii f...": p pointer, i int, l long long,
 * f float). A ctypes call with twenty arguments costs 2.3 us before the launch itself (3 us), this one 0.25.
 *
 * All arguments of integer class go to the callee in their order, in registers and then in 8-byte stack slots, the floats
 * in vector registers in theirs, wherever they stand between the integers (System V x86-64 and Linux AArch64): so one
 * prototype with 32 integers and 4 floats calls every launcher; what it does not read, it does not see.
 *
 * Pointers: an int (tensor.data_ptr()), None (null) or an object with a writable or constant buffer (a ctypes array).
 * Numbers are cut to the declared width as ctypes cuts them. The GIL is released during the call.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#if !(defined(__x86_64__) || defined(__aarch64__)) || !defined(__linux__)
#error "the argument passing below is that of Linux on x86-64 and AArch64"
#endif

#define MAX_INTS 32
#define MAX_FLOATS 4

typedef long long ll;
typedef int (*launcher_fn)(ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll, ll,
                           ll, ll, ll, ll, ll, ll, ll, ll, float, float, float, float);

static long long calls = 0;

typedef struct {
  PyObject_HEAD
  launcher_fn fn;
  int n;
  char sig[MAX_INTS + MAX_FLOATS + 1];
  vectorcallfunc vectorcall;
} Launcher;

/* an integer, or an object that wraps one (ctypes.c_int(5)) */
static int to_int(PyObject* o, ll* out) {
  if (PyLong_Check(o)) {
    *out = (ll)PyLong_AsUnsignedLongLongMask(o);
    return *out == -1 && PyErr_Occurred() ? -1 : 0;
  }
  PyObject* v = PyObject_HasAttrString(o, "value") ? PyObject_GetAttrString(o, "value") : PyNumber_Index(o);
  if (v == NULL) return -1;
  int rc = 0;
  if (v == Py_None) *out = 0;   /* ctypes.c_void_p(0) */
  else {
    PyObject* i = PyNumber_Index(v);
    if (i == NULL) rc = -1;
    else {
      *out = (ll)PyLong_AsUnsignedLongLongMask(i);
      if (*out == -1 && PyErr_Occurred()) rc = -1;
      Py_DECREF(i);
    }
  }
  Py_DECREF(v);
  return rc;
}

static int to_float(PyObject* o, float* out) {
  double d;
  if (PyFloat_Check(o) || PyLong_Check(o) || !PyObject_HasAttrString(o, "value")) {
    d = PyFloat_AsDouble(o);
  } else {
    PyObject* v = PyObject_GetAttrString(o, "value");
    if (v == NULL) return -1;
    d = PyFloat_AsDouble(v);
    Py_DECREF(v);
  }
  if (d == -1.0 && PyErr_Occurred()) return -1;
  *out = (float)d;
  return 0;
}

static PyObject* launcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Launcher* l = (Launcher*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if ((kwnames != NULL && PyTuple_GET_SIZE(kwnames) != 0) || n != l->n)
    return PyErr_Format(PyExc_TypeError, "launcher takes %d positional arguments (%zd given)", l->n, n);
  ll a[MAX_INTS] = {0};
  float f[MAX_FLOATS] = {0};
  Py_buffer views[MAX_INTS];
  int ni = 0, nf = 0, nv = 0, bad = 0;
  for (Py_ssize_t i = 0; i < n && !bad; ++i) {
    PyObject* o = args[i];
    switch (l->sig[i]) {
      case 'f': bad = to_float(o, &f[nf++]); break;
      case 'p':
        if (o == Py_None) {
          a[ni++] = 0;
        } else if (!PyLong_Check(o) && PyObject_CheckBuffer(o) && !PyObject_HasAttrString(o, "value")) {
          bad = PyObject_GetBuffer(o, &views[nv], PyBUF_SIMPLE);
          if (!bad) a[ni++] = (ll)(intptr_t)views[nv++].buf;
        } else {
          bad = to_int(o, &a[ni++]);
        }
        break;
      case 'i': bad = to_int(o, &a[ni]); a[ni] = (int)a[ni]; ++ni; break;
      default: bad = to_int(o, &a[ni++]);
    }
  }
  int rc = 0;
  if (!bad) {
    ++calls;
    Py_BEGIN_ALLOW_THREADS
    rc = l->fn(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16],
               a[17], a[18], a[19], a[20], a[21], a[22], a[23], a[24], a[25], a[26], a[27], a[28], a[29], a[30], a[31], f[0],
               f[1], f[2], f[3]);
    Py_END_ALLOW_THREADS
  }
  for (int i = 0; i < nv; ++i) PyBuffer_Release(&views[i]);
  return bad ? NULL : PyLong_FromLong(rc);
}

static PyObject* launcher_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
  unsigned long long addr;
  const char* sig;
  if (!PyArg_ParseTuple(args, "Ks", &addr, &sig)) return NULL;
  int ni = 0, nf = 0;
  for (const char* c = sig; *c; ++c) {
    if (*c == 'f') ++nf;
    else if (*c == 'p' || *c == 'i' || *c == 'l') ++ni;
    else return PyErr_Format(PyExc_ValueError, "argument type '%c'", *c);
  }
  if (addr == 0 || ni > MAX_INTS || nf > MAX_FLOATS) return PyErr_Format(PyExc_ValueError, "signature %s", sig);
  Launcher* l = (Launcher*)type->tp_alloc(type, 0);
  if (l == NULL) return NULL;
  l->fn = (launcher_fn)(uintptr_t)addr;
  l->n = ni + nf;
  strcpy(l->sig, sig);
  l->vectorcall = launcher_call;
  return (PyObject*)l;
}

static PyTypeObject LauncherType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "_launcher.Launcher",
    .tp_basicsize = sizeof(Launcher),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_new = launcher_new,
    .tp_call = PyVectorcall_Call,
    .tp_vectorcall_offset = offsetof(Launcher, vectorcall),
};

static PyObject* count(PyObject* self, PyObject* none) { return PyLong_FromLongLong(calls); }
static PyMethodDef methods[] = {{"count", count, METH_NOARGS, "calls of all launchers so far"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_launcher", NULL, -1, methods};

PyMODINIT_FUNC PyInit__launcher(void) {
  if (PyType_Ready(&LauncherType) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (m == NULL) return NULL;
  Py_INCREF(&LauncherType);
  if (PyModule_AddObject(m, "Launcher", (PyObject*)&LauncherType) < 0) {
    Py_DECREF(&LauncherType);
    Py_DECREF(m);
    return NULL;
  }
  return m;
}
