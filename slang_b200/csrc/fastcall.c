/* The calls a host loop makes every step, from Python without ctypes: each packs its argument struct and calls the C ABI.
 * A ctypes call with a freshly built argument struct takes 1.5 to 2.5 us, as much as the launch it makes; these take
 * about 0.2.  Every function returns the ABI's code (0, or a negative MLP_E_*). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "../../include/slang_b200_mlp.h"

typedef int32_t (*DispatchFn)(MlpDevice*, MlpKernel*, const void*, size_t, uint32_t, uint32_t, uint32_t);
typedef int32_t (*ClearFn)(MlpDevice*, MlpBuffer*, size_t, size_t);
static DispatchFn g_dispatch;
static ClearFn g_clear;

static int numbers(PyObject* const* args, Py_ssize_t given, Py_ssize_t wanted, uint64_t* out)
{
    if (given != wanted) { PyErr_Format(PyExc_TypeError, "%zd arguments wanted, got %zd", wanted, given); return -1; }
    for (Py_ssize_t i = 0; i < wanted; ++i) {
        out[i] = PyLong_AsUnsignedLongLong(args[i]);
        if (out[i] == (uint64_t)-1 && PyErr_Occurred()) return -1;
    }
    return 0;
}

static PyObject* launch(uint64_t device, uint64_t kernel, const void* args, size_t size, uint64_t groups)
{
    int32_t rc;
    if (groups > 0xffffffffu) { PyErr_SetString(PyExc_OverflowError, "too many groups"); return NULL; }
    Py_BEGIN_ALLOW_THREADS
    rc = g_dispatch((MlpDevice*)device, (MlpKernel*)kernel, args, size, (uint32_t)groups, 1, 1);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static int fits32(uint64_t a, uint64_t b)
{
    if ((a | b) <= 0xffffffffu) return 1;
    PyErr_SetString(PyExc_OverflowError, "counts and flags are 32-bit numbers");
    return 0;
}

/* bind(address of mlp_dispatch, address of mlp_buffer_clear) */
static PyObject* bind(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t v[2];
    if (numbers(args, n, 2, v)) return NULL;
    g_dispatch = (DispatchFn)v[0];
    g_clear = (ClearFn)v[1];
    Py_RETURN_NONE;
}

/* dispatch(device, kernel, struct with a buffer interface, groups) */
static PyObject* dispatch(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t d, k, g;
    Py_buffer b;
    if (n != 4) { PyErr_Format(PyExc_TypeError, "4 arguments wanted, got %zd", n); return NULL; }
    if (numbers(args, 1, 1, &d) || numbers(args + 1, 1, 1, &k) || numbers(args + 3, 1, 1, &g)) return NULL;
    if (PyObject_GetBuffer(args[2], &b, PyBUF_SIMPLE)) return NULL;
    PyObject* r = launch(d, k, b.buf, (size_t)b.len, g);
    PyBuffer_Release(&b);
    return r;
}

/* clear(device, buffer, offset, size) */
static PyObject* clear(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t v[4];
    int32_t rc;
    if (numbers(args, n, 4, v)) return NULL;
    Py_BEGIN_ALLOW_THREADS
    rc = g_clear((MlpDevice*)v[0], (MlpBuffer*)v[1], v[2], v[3]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

/* learn(device, kernel, network, loss, inputs, targets, count, flags, input gradients or 0, groups) */
static PyObject* learn(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t v[10];
    if (numbers(args, n, 10, v) || !fits32(v[6], v[7])) return NULL;
    MlpLearnGradParamsEx2 a = {{v[2], v[3], v[4], v[5], (uint32_t)v[6], (uint32_t)v[7]}, v[8]};
    return launch(v[0], v[1], &a, v[8] ? sizeof a : sizeof a.base, v[9]);
}

/* adjust(device, kernel, states, params, gradients, count, groups) */
static PyObject* adjust(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t v[7];
    if (numbers(args, n, 7, v) || !fits32(v[5], 0)) return NULL;
    MlpAdjustParamsParams a = {v[2], v[3], v[4], (uint32_t)v[5]};
    return launch(v[0], v[1], &a, sizeof a, v[6]);
}

/* forward(device, kernel, network, inputs, outputs, count, flags, groups) */
static PyObject* forward(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    uint64_t v[8];
    if (numbers(args, n, 8, v) || !fits32(v[5], v[6])) return NULL;
    MlpForwardParams a = {v[2], v[3], v[4], (uint32_t)v[5], (uint32_t)v[6]};
    return launch(v[0], v[1], &a, sizeof a, v[7]);
}

static PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, NULL},         {"dispatch", (PyCFunction)(void (*)(void))dispatch, METH_FASTCALL, NULL},
    {"clear", (PyCFunction)(void (*)(void))clear, METH_FASTCALL, NULL},       {"learn", (PyCFunction)(void (*)(void))learn, METH_FASTCALL, NULL},
    {"adjust", (PyCFunction)(void (*)(void))adjust, METH_FASTCALL, NULL},     {"forward", (PyCFunction)(void (*)(void))forward, METH_FASTCALL, NULL},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
