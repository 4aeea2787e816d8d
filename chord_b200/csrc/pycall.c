/* Calls a C-ABI entry point of the library from Python: call(address, signature, arg, ...)
 * with integer arguments, returning its int result.  `signature` has a letter per parameter
 * of the entry point: 'p' a pointer (None is the null pointer), 'i' an integer; another number
 * of arguments is refused.  ctypes does the same at about 4.5 us for the 21 arguments of
 * `indexed` (an argument object each); this takes less than 1 us, on a path that is called once
 * per GEMM.  Every parameter of the entry points it serves is a pointer, an int64_t or an int,
 * which the x86-64 and AArch64 calling conventions pass alike in the registers and eight-byte
 * stack slots of an int64_t; arguments past the callee's last one are ignored by it. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#if !defined(__x86_64__) && !(defined(__aarch64__) && !defined(__APPLE__))
#error "the calling convention assumed here is that of x86-64 and AArch64 Linux"
#endif

enum { kMaxArgs = 24 };

typedef int (*entry_point)(int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                           int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                           int64_t, int64_t, int64_t, int64_t, int64_t, int64_t);

static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t count) {
  (void)self;
  if (count < 2 || !PyUnicode_Check(args[1])) {
    PyErr_SetString(PyExc_TypeError, "call() takes an address, a signature and the entry point's arguments");
    return NULL;
  }
  void* address = PyLong_AsVoidPtr(args[0]);
  if (address == NULL) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry point");
    return NULL;
  }
  Py_ssize_t expected;
  const char* signature = PyUnicode_AsUTF8AndSize(args[1], &expected);
  if (signature == NULL) return NULL;
  if (expected > kMaxArgs || count - 2 != expected) {
    PyErr_Format(PyExc_TypeError, "the entry point takes %zd arguments (at most %d), got %zd", expected, kMaxArgs,
                 count - 2);
    return NULL;
  }
  int64_t a[kMaxArgs] = {0};
  for (Py_ssize_t i = 0; i < expected; ++i) {
    if (args[i + 2] == Py_None && signature[i] == 'p') continue;
    a[i] = PyLong_AsLongLong(args[i + 2]);
    if (a[i] == -1 && PyErr_Occurred()) return NULL;
  }
  int result;
  Py_BEGIN_ALLOW_THREADS
  result = ((entry_point)address)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12],
                                  a[13], a[14], a[15], a[16], a[17], a[18], a[19], a[20], a[21], a[22], a[23]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(result);
}

static PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(address, signature, *arguments) -> int"},
    {NULL, NULL, 0, NULL},
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__call(void) { return PyModule_Create(&module); }
