/* The entry points a decode loop calls over and over, as CPython functions: the same C calls that ctypes makes from the
 * prototypes in _lib.py, without its conversion of every argument through an object. On a B200's host, a call that launches
 * nothing: bi_rms_norm 0.75 -> 0.08 us, bi_matmul 1.43 -> 0.11 us; through the wrappers a norm of one row 9.9 -> 9.0 us, a linear
 * layer of one row, 4096 -> 4096, 19.6 -> 17.0 us.
 * Pointers are integers or None, the interpreter lock is released around the call, the status comes back as an int.
 * bind() takes the functions from the library that _lib.py has loaded. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <stdint.h>
#include "../../include/bi_abi.h"

#define MAX_ARGS 20

/* The arguments by their kinds, a letter each: 'p' a pointer (an address or None), 'i' an integer, 'f' the call's one float.
 * Integers and addresses into v, the float into *f; what the prototype in _lib.py refuses is refused. */
static int take(const char* name, const char* kinds, PyObject* const* args, Py_ssize_t n, Py_ssize_t want, int64_t* v, float* f) {
    if (n != want) {
        PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, want, n);
        return -1;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
        v[i] = 0;
        if (kinds[i] == 'f') {
            *f = (float)PyFloat_AsDouble(args[i]);
        } else if (kinds[i] == 'i') {
            v[i] = PyLong_AsLongLong(args[i]);
            if (v[i] != -1) continue;
        } else if (args[i] != Py_None) {
            v[i] = (int64_t)(intptr_t)PyLong_AsVoidPtr(args[i]);
            if (v[i]) continue;
        }
        if (PyErr_Occurred()) return -1;
    }
    return 0;
}

#define P(i) ((void*)(uintptr_t)v[i])
#define N(i) v[i]
#define Z(i) ((size_t)v[i])
#define I(i) ((int)v[i])
#define ENTRY(NAME, KINDS, ...)                                                                        \
    static __typeof__(NAME)* fn_##NAME;                                                                \
    static PyObject* py_##NAME(PyObject* self, PyObject* const* args, Py_ssize_t n) {                  \
        int64_t v[MAX_ARGS];                                                                           \
        float f = 0.0f;                                                                                \
        int rc;                                                                                        \
        (void)self; (void)f;                                                                           \
        if (!fn_##NAME) { PyErr_SetString(PyExc_RuntimeError, #NAME ": not bound"); return NULL; }      \
        if (take(#NAME, KINDS, args, n, (Py_ssize_t)sizeof(KINDS) - 1, v, &f)) return NULL;             \
        Py_BEGIN_ALLOW_THREADS                                                                         \
        rc = fn_##NAME(__VA_ARGS__);                                                                   \
        Py_END_ALLOW_THREADS                                                                           \
        return PyLong_FromLong(rc);                                                                    \
    }
#define SIZE(NAME, KINDS, ...)                                                                         \
    static __typeof__(NAME)* fn_##NAME;                                                                \
    static PyObject* py_##NAME(PyObject* self, PyObject* const* args, Py_ssize_t n) {                  \
        int64_t v[MAX_ARGS];                                                                           \
        float f;                                                                                       \
        (void)self;                                                                                    \
        if (!fn_##NAME) { PyErr_SetString(PyExc_RuntimeError, #NAME ": not bound"); return NULL; }      \
        if (take(#NAME, KINDS, args, n, (Py_ssize_t)sizeof(KINDS) - 1, v, &f)) return NULL;             \
        return PyLong_FromSize_t(fn_##NAME(__VA_ARGS__));                                              \
    }

ENTRY(bi_rms_norm, "pppiifip", P(0), P(1), P(2), N(3), N(4), f, I(6), P(7))
ENTRY(bi_add_rms_norm, "pppppiifip", P(0), P(1), P(2), P(3), P(4), N(5), N(6), f, I(8), P(9))
ENTRY(bi_matmul, "ppppiiiiiiiiiipp", P(0), P(1), P(2), P(3), Z(4), N(5), N(6), N(7), N(8), N(9), N(10), N(11), I(12), I(13), P(14), P(15))
ENTRY(bi_matmul_bias, "pppppiiiiiiiiiipp", P(0), P(1), P(2), P(3), P(4), Z(5), N(6), N(7), N(8), N(9), N(10), N(11), N(12), I(13), I(14), P(15), P(16))
ENTRY(bi_qmm, "ppppppiiiiiiiiipp", P(0), P(1), P(2), P(3), P(4), P(5), Z(6), N(7), N(8), N(9), N(10), I(11), I(12), I(13), I(14), P(15), P(16))
ENTRY(bi_attn_decode, "ppppppiiiiiiiiifiip", P(0), P(1), P(2), P(3), P(4), P(5), Z(6), N(7), N(8), N(9), N(10), N(11), N(12), N(13), N(14), f, I(16), I(17), P(18))
ENTRY(bi_attn_prefill, "ppppiiiiiiiiifiiip", P(0), P(1), P(2), P(3), N(4), N(5), N(6), N(7), N(8), N(9), N(10), N(11), N(12), f, I(14), I(15), I(16), P(17))
SIZE(bi_matmul_scratch_bytes, "iiii", N(0), N(1), N(2), I(3))
SIZE(bi_qmm_scratch_bytes, "iiii", N(0), N(1), N(2), I(3))
SIZE(bi_attn_decode_workspace_bytes, "iiiii", N(0), N(1), N(2), N(3), I(4))

static PyObject* py_bind(PyObject* self, PyObject* handle) {
    void* h = PyLong_AsVoidPtr(handle);
    (void)self;
    if (PyErr_Occurred()) return NULL;
#define BIND(NAME)                                                                                     \
    fn_##NAME = (__typeof__(fn_##NAME))dlsym(h, #NAME);                                                \
    if (!fn_##NAME) { PyErr_SetString(PyExc_RuntimeError, "the kernel library has no " #NAME); return NULL; }
    BIND(bi_rms_norm) BIND(bi_add_rms_norm) BIND(bi_matmul) BIND(bi_matmul_bias) BIND(bi_qmm) BIND(bi_attn_decode)
    BIND(bi_attn_prefill) BIND(bi_matmul_scratch_bytes) BIND(bi_qmm_scratch_bytes) BIND(bi_attn_decode_workspace_bytes)
    Py_RETURN_NONE;
}

#define METHOD(NAME) {#NAME, (PyCFunction)(void (*)(void))py_##NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    METHOD(bi_rms_norm), METHOD(bi_add_rms_norm), METHOD(bi_matmul), METHOD(bi_matmul_bias), METHOD(bi_qmm),
    METHOD(bi_attn_decode), METHOD(bi_attn_prefill), METHOD(bi_matmul_scratch_bytes), METHOD(bi_qmm_scratch_bytes),
    METHOD(bi_attn_decode_workspace_bytes), {"bind", py_bind, METH_O, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&module); }
