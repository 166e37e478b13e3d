// Calls into the C-ABI for capi.py's hot entry points.
//
// A C-ABI call through ctypes costs 0.8-1.2 us for its argument conversions,
// and an array of NTT handles 0.2 us per handle, against 2-3 us for the
// launches behind it: a third of a small transform's host time.  call() passes
// up to 14 integers (System V: every argument of these functions is an
// integer or pointer of at most 64 bits in a register or 8-byte stack slot).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#define MAX_ARGS 14
#define MAX_ITEMS 256

typedef int32_t (*fn_t)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

static PyObject* s_hv;  // attribute of NTT: its handle's address as an int

static int as_u64(PyObject* o, uint64_t* out)
{
    if (o == Py_None) {
        *out = 0;
        return 0;
    }
    if (!PyLong_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected an integer, got %.100s", Py_TYPE(o)->tp_name);
        return -1;
    }
    *out = PyLong_AsUnsignedLongLongMask(o);
    return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
}

// call(address, *args) -> status.  An argument is an int, None (0), or a list
// or tuple of ints or of NTT objects, passed as the address of an array of
// their values, with an element count the caller passes itself.
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t nargs)
{
    (void)self;
    uint64_t a[MAX_ARGS] = {0}, items[MAX_ITEMS], addr;
    uint64_t* heap[MAX_ARGS] = {0};
    Py_ssize_t used = 0;
    PyObject* ret = NULL;
    if (nargs < 1 || nargs > MAX_ARGS + 1) {
        PyErr_SetString(PyExc_TypeError, "call(address, up to 14 arguments)");
        return NULL;
    }
    if (as_u64(args[0], &addr)) return NULL;
    for (Py_ssize_t i = 1; i < nargs; ++i) {
        PyObject* o = args[i];
        if (!PyList_Check(o) && !PyTuple_Check(o)) {
            if (as_u64(o, &a[i - 1])) goto done;
            continue;
        }
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
        uint64_t* to = items + used;
        if (n > MAX_ITEMS - used) {
            to = heap[i - 1] = PyMem_Malloc((size_t)n * sizeof(uint64_t));
            if (!to) {
                PyErr_NoMemory();
                goto done;
            }
        } else {
            used += n;
        }
        for (Py_ssize_t k = 0; k < n; ++k) {
            if (k >= PySequence_Fast_GET_SIZE(o)) {  // an attribute lookup below may run Python code
                PyErr_SetString(PyExc_RuntimeError, "list changed during the call");
                goto done;
            }
            PyObject* e = PySequence_Fast_GET_ITEM(o, k);
            if (PyLong_Check(e) || e == Py_None) {
                if (as_u64(e, &to[k])) goto done;
            } else {
                PyObject* v = PyObject_GetAttr(e, s_hv);
                if (!v) goto done;
                const int bad = as_u64(v, &to[k]);
                Py_DECREF(v);
                if (bad) goto done;
            }
        }
        a[i - 1] = (uint64_t)(uintptr_t)to;
    }
    int32_t st;
    Py_BEGIN_ALLOW_THREADS
    st = ((fn_t)(uintptr_t)addr)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12],
                                 a[13]);
    Py_END_ALLOW_THREADS
    ret = PyLong_FromLong(st);
done:
    for (int i = 0; i < MAX_ARGS; ++i) PyMem_Free(heap[i]);
    return ret;
}

static PyMethodDef methods[] = {{"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(address, *args) -> status"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void)
{
    s_hv = PyUnicode_InternFromString("hv");
    return s_hv ? PyModule_Create(&module) : NULL;
}
