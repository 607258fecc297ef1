// Calls of the C ABI from Python without ctypes' conversions: bind(address, "argument types", "result type", slow) gives a callable that
// passes integers, None, bytes (their address) and floats straight on.  Anything else (a ctypes object, a wrong number of
// arguments) goes to `slow`, the ctypes function for the same entry, which takes or refuses it as ever.
//
// Types: p pointer, i 32-bit and l 64-bit integer, f float; the result i, z (size_t).  Integers are cut to their width without a
// check, as ctypes does.  Only for the x86-64 System V calling convention: integers and floats are counted there separately, so the
// order between the two does not matter, and an integer narrower than a register may come with anything above it.
// Passing on the 19 arguments of a decode takes 0.2 us, 2.2 through ctypes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "argument passing is that of x86-64 System V"
#endif

enum { kMaxArgs = 28, kMaxFloats = 4 };

typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    void* address;
    PyObject* slow;
    int n;
    char result;
    char types[kMaxArgs + 1];
} Call;

typedef int64_t W;
// Every argument that a function does not have is passed all the same: the caller clears the stack, nobody reads it.
typedef W (*Fn)(W, W, W, W, W, W, float, float, float, float, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W);

static PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
    Call* c = (Call*)self;
    const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
    W w[kMaxArgs] = {0};
    float f[kMaxFloats] = {0};
    int nw = 0, nf = 0;
    if (n != c->n || kwnames != NULL) return PyObject_Vectorcall(c->slow, args, nargsf, kwnames);
    for (Py_ssize_t k = 0; k < n; ++k) {
        PyObject* const a = args[k];
        if (c->types[k] == 'f') {
            double d;
            if (PyFloat_CheckExact(a)) d = PyFloat_AS_DOUBLE(a);
            else if (PyLong_Check(a)) d = PyLong_AsDouble(a);
            else return PyObject_Vectorcall(c->slow, args, nargsf, kwnames);
            if (d == -1.0 && PyErr_Occurred()) return NULL;
            f[nf++] = (float)d;
        } else if (PyLong_Check(a)) {
            w[nw++] = (W)PyLong_AsUnsignedLongLongMask(a);
        } else if (c->types[k] == 'p' && a == Py_None) {
            w[nw++] = 0;
        } else if (c->types[k] == 'p' && PyBytes_CheckExact(a)) {
            w[nw++] = (W)(uintptr_t)PyBytes_AS_STRING(a);
        } else {
            return PyObject_Vectorcall(c->slow, args, nargsf, kwnames);
        }
    }
    W r;
    const Fn fn = (Fn)c->address;
    Py_BEGIN_ALLOW_THREADS
    r = fn(w[0], w[1], w[2], w[3], w[4], w[5], f[0], f[1], f[2], f[3], w[6], w[7], w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15], w[16], w[17],
           w[18], w[19], w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27]);
    Py_END_ALLOW_THREADS
    return c->result == 'i' ? PyLong_FromLong((int32_t)r) : PyLong_FromSize_t((size_t)r);
}

static void dealloc(PyObject* self) {
    Py_XDECREF(((Call*)self)->slow);
    Py_TYPE(self)->tp_free(self);
}

static PyTypeObject CallType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "b2kv_calls.Call",
    .tp_basicsize = sizeof(Call),
    .tp_dealloc = dealloc,
    .tp_vectorcall_offset = offsetof(Call, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
};

static PyObject* bind(PyObject* module, PyObject* args) {
    unsigned long long address;
    const char *types, *result;
    PyObject* slow;
    (void)module;
    if (!PyArg_ParseTuple(args, "KssO", &address, &types, &result, &slow)) return NULL;
    size_t n = strlen(types), floats = 0;
    for (size_t k = 0; k < n; ++k) {
        if (strchr("pilf", types[k]) == NULL) return PyErr_Format(PyExc_ValueError, "unknown argument type in %s", types);
        floats += types[k] == 'f';
    }
    if (n > kMaxArgs || floats > kMaxFloats || (strcmp(result, "i") != 0 && strcmp(result, "z") != 0))
        return PyErr_Format(PyExc_ValueError, "no such call: %s -> %s", types, result);
    Call* c = PyObject_New(Call, &CallType);
    if (c == NULL) return NULL;
    c->vectorcall = call;
    c->address = (void*)(uintptr_t)address;
    Py_INCREF(slow);
    c->slow = slow;
    c->n = (int)n;
    c->result = result[0];
    memcpy(c->types, types, n + 1);
    return (PyObject*)c;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "b2kv_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_b2kv_calls(void) {
    if (PyType_Ready(&CallType) < 0) return NULL;
    return PyModule_Create(&module);
}
