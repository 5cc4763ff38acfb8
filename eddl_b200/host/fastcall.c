/* Native caller of the C ABI for Python: `call(name, *args)` of eddl_b200.capi without ctypes on the way.
 *
 * A pass over a small net is a few dozen calls of this library, and the ctypes conversion of up to twenty arguments costs
 * more than the call itself (3.4 us for conv2d_fwd, plus 1.1 us to look for DeviceArrays among the arguments).  The wrappers
 * in fastcall_table.inc, one per function declared in include/eddl_b200.h, are generated from that header when the library
 * is built, so they cannot drift from the declarations.  They take what ctypes takes for the same parameter -- None, an
 * int, a DeviceArray, a ctypes array (its address) for a pointer, an int for an integer, a float or int for a float -- and
 * integers wrap around as they do there; for anything else (byref(), bytes, c_void_p objects, wrong counts) the wrapper
 * answers "not mine" and the ctypes path of the binding runs the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include "eddl_b200.h"

static PyTypeObject *g_device_array, *g_ctypes_array;
static PyObject *g_addr, *g_slow, *g_fail;

static inline int to_int(PyObject *o, int *v) {
    if (!PyLong_CheckExact(o)) return 0;
    *v = (int)PyLong_AsUnsignedLongMask(o);
    return 1;
}
static inline int to_size(PyObject *o, size_t *v) {
    if (!PyLong_CheckExact(o)) return 0;
    *v = (size_t)PyLong_AsUnsignedLongLongMask(o);
    return 1;
}
static inline int to_float(PyObject *o, float *v) {
    if (PyFloat_CheckExact(o)) { *v = (float)PyFloat_AS_DOUBLE(o); return 1; }
    if (!PyLong_CheckExact(o)) return 0;
    const double d = PyLong_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
    *v = (float)d;
    return 1;
}
static int to_ptr(PyObject *o, void **v) {
    if (o == Py_None) { *v = NULL; return 1; }
    if (PyLong_CheckExact(o)) { *v = (void *)(uintptr_t)PyLong_AsUnsignedLongLongMask(o); return 1; }
    if (PyObject_TypeCheck(o, g_device_array)) {
        PyObject *a = PyObject_GetAttr(o, g_addr);
        int ok = a && PyLong_CheckExact(a);
        if (ok) *v = (void *)(uintptr_t)PyLong_AsUnsignedLongLongMask(a);
        Py_XDECREF(a);
        if (!ok) PyErr_Clear();
        return ok;
    }
    if (PyObject_TypeCheck(o, g_ctypes_array)) {
        Py_buffer b;
        if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) { PyErr_Clear(); return 0; }
        *v = b.buf;
        PyBuffer_Release(&b);           /* the caller's tuple keeps the array, and with it the memory, alive */
        return 1;
    }
    return 0;
}

typedef int (*Wrapper)(PyObject *const *a, Py_ssize_t n, int *status);     /* 0 = not mine */
#include "fastcall_table.inc"

static PyObject *g_index;               /* name -> position in the table */

static PyObject *call(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    (void)self;
    if (n >= 1) {
        PyObject *at = PyDict_GetItemWithError(g_index, args[0]);
        if (at) {
            int status = 0;
            if (g_table[PyLong_AsSsize_t(at)].fn(args + 1, n - 1, &status)) {
                if (status == 0) Py_RETURN_NONE;
                return PyObject_CallFunction(g_fail, "Oi", args[0], status);
            }
        } else if (PyErr_Occurred()) PyErr_Clear();
    }
    return PyObject_Vectorcall(g_slow, args, (size_t)n, NULL);
}

/* setup(DeviceArray, ctypes.Array, slow, fail) */
static PyObject *setup(PyObject *self, PyObject *args) {
    (void)self;
    PyObject *d, *c, *s, *f;
    if (!PyArg_ParseTuple(args, "O!O!OO", &PyType_Type, &d, &PyType_Type, &c, &s, &f)) return NULL;
    Py_INCREF(d); Py_INCREF(c); Py_INCREF(s); Py_INCREF(f);
    g_device_array = (PyTypeObject *)d; g_ctypes_array = (PyTypeObject *)c; g_slow = s; g_fail = f;
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(name, *args): one function of the C ABI"},
    {"setup", setup, METH_VARARGS, "setup(DeviceArray, ctypes.Array, slow, fail)"},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
    g_addr = PyUnicode_InternFromString("addr");
    g_index = PyDict_New();
    if (!g_addr || !g_index) return NULL;
    for (Py_ssize_t i = 0; g_table[i].name; i++) {
        PyObject *k = PyUnicode_InternFromString(g_table[i].name), *v = PyLong_FromSsize_t(i);
        if (!k || !v || PyDict_SetItem(g_index, k, v) != 0) return NULL;
        Py_DECREF(k); Py_DECREF(v);
    }
    return PyModule_Create(&module);
}
