// Calls into the C-ABI for capi.py's hot entry points.
//
// A C-ABI call through ctypes costs 0.8-1.2 us for its argument conversions,
// and an array of NTT handles 0.2 us per handle, against 2-3 us for the
// launches behind it: a third of a small transform's host time.  A callable
// made by entry() passes up to 14 integers (System V: every argument of these functions is an
// integer or pointer of at most 64 bits in a register or 8-byte stack slot).
//
// It converts the plain argument forms only, each as ctypes converts it, and
// answers None without a call for any other, which capi.py then gives to
// ctypes: what is taken and what is refused is ctypes' decision.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#define MAX_ARGS 14
#define MAX_ITEMS 256

typedef int32_t (*fn_t)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                        uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

static PyObject* s_hv;      // attribute of NTT: its handle's address as an int
static PyObject* ntt_type;  // capi.NTT

// 1: converted, 0: another form, -1: error.
static int from_int(PyObject* o, uint64_t* out)
{
    if (!PyLong_Check(o)) return 0;
    *out = PyLong_AsUnsignedLongLongMask(o);
    return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 1;
}

// An integer parameter: anything with __index__, as for a c_uint64.
static int from_index(PyObject* o, uint64_t* out)
{
    if (PyLong_Check(o)) return from_int(o, out);
    if (!PyIndex_Check(o)) return 0;
    PyObject* v = PyNumber_Index(o);
    if (!v) {
        PyErr_Clear();
        return 0;
    }
    const int r = from_int(v, out);
    Py_DECREF(v);
    return r;
}

// An address: an int, or None for null, as for a c_void_p.
static int from_address(PyObject* o, uint64_t* out)
{
    if (o != Py_None) return from_int(o, out);
    *out = 0;
    return 1;
}

// The address of an NTT object's handle.
static int from_ntt(PyObject* o, uint64_t* out)
{
    if (!ntt_type || !PyObject_TypeCheck(o, (PyTypeObject*)ntt_type)) return 0;
    PyObject* v = PyObject_GetAttr(o, s_hv);
    if (!v) {
        PyErr_Clear();
        return 0;
    }
    const int r = from_int(v, out);
    Py_DECREF(v);
    return r;
}

// What an entry point's callable carries: its address and one letter per
// argument, "i" an integer, "p" an address, "h" a list or tuple of NTT objects
// and "a" one of ints, these two passed as the address of an array of their
// values (the caller passes their count too).
typedef struct {
    fn_t fn;
    int len;
    char kinds[MAX_ARGS];
} entry_t;

// (*args) -> status, or None if an argument has another form.
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t nargs)
{
    const entry_t* entry = PyCapsule_GetPointer(self, NULL);
    uint64_t a[MAX_ARGS] = {0}, items[MAX_ITEMS];
    uint64_t* heap[MAX_ARGS] = {0};
    Py_ssize_t used = 0;
    if (!entry) return NULL;
    const Py_ssize_t len = entry->len;
    if (nargs != len) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", len, nargs);
        return NULL;
    }
    int r = 1;
    for (Py_ssize_t i = 0; r == 1 && i < len; ++i) {
        PyObject* o = args[i];
        const char kind = entry->kinds[i];
        if (kind == 'i') {
            r = from_index(o, &a[i]);
            continue;
        }
        if (kind == 'p') {
            r = from_address(o, &a[i]);
            continue;
        }
        if (!PyList_Check(o) && !PyTuple_Check(o)) {
            r = 0;
            break;
        }
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
        uint64_t* to = items + used;
        if (n > MAX_ITEMS - used) {
            to = heap[i] = PyMem_Malloc((size_t)n * sizeof(uint64_t));
            if (!to) {
                PyErr_NoMemory();
                r = -1;
                break;
            }
        } else {
            used += n;
        }
        for (Py_ssize_t k = 0; r == 1 && k < n; ++k) {
            if (k >= PySequence_Fast_GET_SIZE(o)) {  // an attribute lookup may run Python code
                PyErr_SetString(PyExc_RuntimeError, "list changed during the call");
                r = -1;
                break;
            }
            PyObject* e = PySequence_Fast_GET_ITEM(o, k);
            Py_INCREF(e);
            r = kind == 'h' ? from_ntt(e, &to[k]) : from_int(e, &to[k]);
            Py_DECREF(e);
        }
        a[i] = (uint64_t)(uintptr_t)to;
    }
    PyObject* ret = NULL;
    if (r == 1) {
        int32_t st;
        Py_BEGIN_ALLOW_THREADS
        st = entry->fn(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13]);
        Py_END_ALLOW_THREADS
        ret = PyLong_FromLong(st);
    } else if (r == 0) {
        ret = Py_NewRef(Py_None);
    }
    for (int i = 0; i < MAX_ARGS; ++i) PyMem_Free(heap[i]);
    return ret;
}

static PyMethodDef call_def = {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL,
                               "(*args) -> status, or None if an argument has another form"};

static void free_entry(PyObject* capsule) { PyMem_Free(PyCapsule_GetPointer(capsule, NULL)); }

// entry(address, kinds): the callable of an entry point.
static PyObject* entry(PyObject* self, PyObject* args)
{
    (void)self;
    unsigned long long address;
    const char* kinds;
    Py_ssize_t len;
    if (!PyArg_ParseTuple(args, "Ks#", &address, &kinds, &len)) return NULL;
    if (len > MAX_ARGS) {
        PyErr_SetString(PyExc_ValueError, "too many arguments");
        return NULL;
    }
    entry_t* e = PyMem_Malloc(sizeof *e);
    if (!e) return PyErr_NoMemory();
    e->fn = (fn_t)(uintptr_t)address;
    e->len = (int)len;
    memcpy(e->kinds, kinds, (size_t)len);
    PyObject* capsule = PyCapsule_New(e, NULL, free_entry);
    if (!capsule) {
        PyMem_Free(e);
        return NULL;
    }
    PyObject* f = PyCFunction_NewEx(&call_def, capsule, NULL);
    Py_DECREF(capsule);
    return f;
}

// handle_type(cls): the class whose objects an "h" list holds.
static PyObject* handle_type(PyObject* self, PyObject* cls)
{
    (void)self;
    if (!PyType_Check(cls)) {
        PyErr_SetString(PyExc_TypeError, "expected a class");
        return NULL;
    }
    Py_XSETREF(ntt_type, Py_NewRef(cls));
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"entry", entry, METH_VARARGS, "entry(address, kinds) -> callable"},
    {"handle_type", handle_type, METH_O, "handle_type(cls)"},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void)
{
    s_hv = PyUnicode_InternFromString("hv");
    return s_hv ? PyModule_Create(&module) : NULL;
}
