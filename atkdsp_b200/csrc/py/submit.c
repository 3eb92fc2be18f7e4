/* Server.submit's argument work as a CPython module. A round of many small
 * streams is one call per block, and through ctypes each took 2.4 us (two
 * pointer objects, eight conversions, the GIL dropped and taken again); from
 * here it takes 0.6. A round of 256 streams, whose launch runs 0.2 ms, went
 * from 795 to 468 us. The library's function is passed in by address, so the
 * module links against nothing and serves whichever library was loaded. */
#define Py_LIMITED_API 0x030C0000          /* one build serves Python 3.12 and later */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#if PY_VERSION_HEX < 0x030C0000
#error "needs Python 3.12's headers: PyObject_VectorcallMethod is outside the limited API before"
#endif

typedef int (*submit_fn)(void *s, int id, const void *d_raw, size_t n, void *d_out, size_t cap, uint64_t tag,
                         double t_arrival);

static PyObject *s_numel, *s_data_ptr, *s_dtype;

/* o as int(o) does, then the low 64 bits, as ctypes converts integers */
static int as_u64(PyObject *o, uint64_t *v) {
    PyObject *l = PyNumber_Long(o);
    if (!l) return 0;
    *v = (uint64_t)PyLong_AsUnsignedLongLongMask(l);
    Py_DECREF(l);
    return *v != (uint64_t)-1 || !PyErr_Occurred();
}

static int method_u64(PyObject *o, PyObject *name, uint64_t *v) {
    PyObject *r = PyObject_VectorcallMethod(name, &o, 1, NULL);
    if (!r) return 0;
    const int ok = as_u64(r, v);
    Py_DECREF(r);
    return ok;
}

/* submit(fn, server, cf32_dtype, sid, block, out, tag, t_arrival) -> int */
static PyObject *submit(PyObject *self, PyObject *const *a, Py_ssize_t n_args) {
    uint64_t fn, srv, sid, raw, n, out, cap, tag;
    (void)self;
    if (n_args != 8) {
        PyErr_SetString(PyExc_TypeError, "submit takes 8 arguments");
        return NULL;
    }
    PyObject *block = a[4], *dt = PyObject_GetAttr(block, s_dtype);
    if (!dt) return NULL;
    const int cf32 = PyObject_RichCompareBool(dt, a[2], Py_EQ);
    Py_DECREF(dt);
    if (cf32 < 0 || !method_u64(block, s_numel, &n)) return NULL;
    if (!cf32) n /= 2;
    if (!as_u64(a[0], &fn) || !as_u64(a[1], &srv) || !as_u64(a[3], &sid) || !method_u64(block, s_data_ptr, &raw) ||
        !method_u64(a[5], s_data_ptr, &out) || !method_u64(a[5], s_numel, &cap) || !as_u64(a[6], &tag))
        return NULL;
    PyObject *t = PyNumber_Float(a[7]);
    if (!t) return NULL;
    const double at = PyFloat_AsDouble(t);
    Py_DECREF(t);
    const int rc = ((submit_fn)(uintptr_t)fn)((void *)(uintptr_t)srv, (int)(uint32_t)sid,
                                              (const void *)(uintptr_t)raw, (size_t)n, (void *)(uintptr_t)out,
                                              (size_t)cap, tag, at);
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"submit", (PyCFunction)(void (*)(void))submit, METH_FASTCALL,
                                 "atkdsp_server_submit of a block tensor into an output tensor"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef def = {PyModuleDef_HEAD_INIT, "_atkdsp_submit", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__atkdsp_submit(void) {
    s_numel = PyUnicode_InternFromString("numel");
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_dtype = PyUnicode_InternFromString("dtype");
    if (!s_numel || !s_data_ptr || !s_dtype) return NULL;
    return PyModule_Create(&def);
}
