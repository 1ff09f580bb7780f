// CPython entry for the calls whose device work takes a few microseconds (a decode step's linears): ctypes spends about
// 1.2 us per call on building pointer objects and converting six arguments, this 0.2.
//
//   call6(function address, ctx, w, x, M, C, ldc) -> status      int f(void *, const void *, const void *, int, void *, int)
//
// The function is one of libinkq.so's, loaded by the package; this module links against nothing of it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

typedef int (*Call6)(void *, const void *, const void *, int, void *, int);

static PyObject *call6(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    if (n != 7) {
        PyErr_SetString(PyExc_TypeError, "call6 takes seven integers");
        return NULL;
    }
    unsigned long long p[5];
    static const int at[5] = {0, 1, 2, 3, 5};
    for (int i = 0; i < 5; i++) {
        p[i] = PyLong_AsUnsignedLongLong(args[at[i]]);
        if (p[i] == static_cast<unsigned long long>(-1) && PyErr_Occurred()) return NULL;
    }
    const long M = PyLong_AsLong(args[4]), ldc = PyLong_AsLong(args[6]);
    if ((M == -1 || ldc == -1) && PyErr_Occurred()) return NULL;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = reinterpret_cast<Call6>(p[0])(reinterpret_cast<void *>(p[1]), reinterpret_cast<const void *>(p[2]), reinterpret_cast<const void *>(p[3]),
                                       static_cast<int>(M), reinterpret_cast<void *>(p[4]), static_cast<int>(ldc));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"call6", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(call6)), METH_FASTCALL, "call6(fn, ctx, w, x, M, C, ldc)"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "inkq_fast_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_inkq_fast_call(void) { return PyModule_Create(&module); }
