/* Calls from Python into the kernel library's C interface without ctypes' conversion of every argument (about 0.1 us each, 20 to
 * 45 arguments a call, which for steps of few tokens is a fifth of the time a launch takes the host).
 *
 * bind(address, signature) -> callable.  signature: a letter an argument, 'p' an address (an integer or None), 'i' an integer of
 * any width, 'f' a float.  The function must return int.  The callable releases the interpreter lock during the call, as ctypes
 * does, and returns the function's result; or NotImplemented, without having called, when an argument is of another kind (an
 * array, a reference to a structure): the caller then goes through ctypes.
 *
 * How one call serves every signature: in the System V calling convention of x86-64 integers and addresses take six registers
 * and then eight-byte places on the stack, in their order among themselves, floats take registers of their own (up to eight), and
 * the caller clears the stack.  So a function may be called with all its integers first, its floats behind them, and more of
 * either than it has.  14 arguments: 2.2 us through ctypes, 0.23 us here. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "the universal call relies on the System V calling convention of x86-64"
#endif

#define MAX_INTS 64
#define MAX_FLOATS 8
#define I8(k) a[k], a[k + 1], a[k + 2], a[k + 3], a[k + 4], a[k + 5], a[k + 6], a[k + 7]
#define L8 long, long, long, long, long, long, long, long

typedef int (*universal)(L8, L8, L8, L8, L8, L8, L8, L8, float, float, float, float, float, float, float, float);

typedef struct {
  universal fn;
  Py_ssize_t n;
  char sig[128];
} entry;

static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  const entry* e = (const entry*)PyCapsule_GetPointer(self, "lb_caller.entry");
  if (!e) return NULL;
  if (nargs != e->n) {
    PyErr_Format(PyExc_TypeError, "this function takes %zd arguments (%zd given)", e->n, nargs);
    return NULL;
  }
  long a[MAX_INTS];
  float f[MAX_FLOATS] = {0};
  int ni = 0, nf = 0;
  for (Py_ssize_t i = 0; i < nargs; ++i) {
    PyObject* x = args[i];
    if (e->sig[i] == 'f') {
      if (PyFloat_Check(x)) f[nf++] = (float)PyFloat_AS_DOUBLE(x);
      else if (PyLong_Check(x)) {
        const double d = PyLong_AsDouble(x);
        if (d == -1.0 && PyErr_Occurred()) return NULL;
        f[nf++] = (float)d;
      } else Py_RETURN_NOTIMPLEMENTED;
    } else if (PyLong_Check(x)) {
      int overflow = 0;
      long long v = PyLong_AsLongLongAndOverflow(x, &overflow);
      if (overflow > 0) v = (long long)PyLong_AsUnsignedLongLongMask(x);       /* an address or key above 2^63 */
      else if (overflow < 0) Py_RETURN_NOTIMPLEMENTED;
      a[ni++] = (long)v;
    } else if (e->sig[i] == 'p' && x == Py_None) {
      a[ni++] = 0;
    } else {
      Py_RETURN_NOTIMPLEMENTED;
    }
  }
  while (ni < MAX_INTS) a[ni++] = 0;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = e->fn(I8(0), I8(8), I8(16), I8(24), I8(32), I8(40), I8(48), I8(56), f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMethodDef call_def = {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, NULL};

static void drop(PyObject* capsule) { PyMem_Free(PyCapsule_GetPointer(capsule, "lb_caller.entry")); }

static PyObject* bind(PyObject* self, PyObject* args) {
  (void)self;
  unsigned long long address;
  const char* sig;
  Py_ssize_t n;
  if (!PyArg_ParseTuple(args, "Ks#", &address, &sig, &n)) return NULL;
  int ni = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (sig[i] == 'f') ++nf;
    else if (sig[i] == 'p' || sig[i] == 'i') ++ni;
    else return PyErr_Format(PyExc_ValueError, "signature letter %c", sig[i]);
  }
  if (!address || n >= 128 || ni > MAX_INTS || nf > MAX_FLOATS) return PyErr_Format(PyExc_ValueError, "no address, or too many arguments");
  entry* e = (entry*)PyMem_Calloc(1, sizeof(entry));
  if (!e) return PyErr_NoMemory();
  e->fn = (universal)(uintptr_t)address;
  e->n = n;
  memcpy(e->sig, sig, (size_t)n);
  PyObject* capsule = PyCapsule_New(e, "lb_caller.entry", drop);
  if (!capsule) { PyMem_Free(e); return NULL; }
  PyObject* f = PyCFunction_NewEx(&call_def, capsule, NULL);
  Py_DECREF(capsule);
  return f;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(address, signature) -> callable"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "lb_caller", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit_lb_caller(void) { return PyModule_Create(&module); }
