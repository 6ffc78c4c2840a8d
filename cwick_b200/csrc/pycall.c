/* pycall.c -- the entry points of a decode step as CPython functions.
 *
 * The same calls through ctypes cost 2.4 us each in argument conversion, as much as a kernel launch, and a decode step at
 * small batch is bound by what the host spends per call. Arguments are those of include/cwk_attn.h in their order: pointers
 * as integers (tensor.data_ptr()) or None, sizes as integers, scales as floats. Each returns the status. The calls run
 * without the interpreter lock, as through ctypes. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/cwk_attn.h"

static void *ptr(PyObject *o) { return o == Py_None ? NULL : (void *)(uintptr_t)PyLong_AsUnsignedLongLong(o); }
static int64_t i64(PyObject *o) { return (int64_t)PyLong_AsLongLong(o); }
static int i32(PyObject *o) { return (int)PyLong_AsLong(o); }
static float f32(PyObject *o) { return (float)PyFloat_AsDouble(o); }

#define WRAP(name, count, ...)                                                                               \
    static PyObject *py_##name(PyObject *self, PyObject *const *a, Py_ssize_t n) {                          \
        (void)self;                                                                                          \
        if (n != (count)) return PyErr_Format(PyExc_TypeError, #name " takes %d arguments", (int)(count)); \
        __VA_ARGS__                                                                                          \
    }
#define RUN(expr)                       \
    do {                                \
        int s;                          \
        if (PyErr_Occurred()) return NULL; \
        Py_BEGIN_ALLOW_THREADS          \
        s = (expr);                     \
        Py_END_ALLOW_THREADS            \
        return PyLong_FromLong(s);      \
    } while (0)

WRAP(cwk_mla_decode, 16, {
    cwk_ctx *c = ptr(a[0]); void *q = ptr(a[1]), *cache = ptr(a[2]); const int64_t stride = i64(a[3]), ld = i64(a[4]);
    void *len = ptr(a[5]); const int max_len = i32(a[6]); void *sel = ptr(a[7]); const int64_t sel_ld = i64(a[8]);
    const int B = i32(a[9]), nh = i32(a[10]), L = i32(a[11]), R = i32(a[12]); const float scale = f32(a[13]);
    void *out = ptr(a[14]); const int splits = i32(a[15]);
    RUN(cwk_mla_decode(c, q, cache, stride, ld, len, max_len, sel, sel_ld, B, nh, L, R, scale, out, splits));
})
WRAP(cwk_gqa_decode, 14, {
    cwk_ctx *c = ptr(a[0]); void *q = ptr(a[1]), *k = ptr(a[2]), *v = ptr(a[3]); const int64_t stride = i64(a[4]);
    void *len = ptr(a[5]); const int max_len = i32(a[6]), B = i32(a[7]), nh = i32(a[8]), nkv = i32(a[9]), hd = i32(a[10]);
    const float scale = f32(a[11]); void *out = ptr(a[12]); const int splits = i32(a[13]);
    RUN(cwk_gqa_decode(c, q, k, v, stride, len, max_len, B, nh, nkv, hd, scale, out, splits));
})
WRAP(cwk_dsa_select, 17, {
    cwk_ctx *c = ptr(a[0]); void *keys = ptr(a[1]), *ks = ptr(a[2]); const int64_t stride = i64(a[3]);
    void *q = ptr(a[4]), *wt = ptr(a[5]), *len = ptr(a[6]); const int max_n = i32(a[7]), B = i32(a[8]), ih = i32(a[9]), hd = i32(a[10]);
    const int want = i32(a[11]), self_ = i32(a[12]); void *sel = ptr(a[13]); const int64_t sel_ld = i64(a[14]);
    void *nsel = ptr(a[15]), *scores = ptr(a[16]);
    RUN(cwk_dsa_select(c, keys, ks, stride, q, wt, len, max_n, B, ih, hd, want, self_, sel, sel_ld, nsel, scores));
})
WRAP(cwk_gdn_scan, 17, {
    cwk_ctx *c = ptr(a[0]); const int B = i32(a[1]), n_ = i32(a[2]), nh = i32(a[3]), hk = i32(a[4]), hv = i32(a[5]), grp = i32(a[6]);
    void *up = ptr(a[7]), *gd = ptr(a[8]), *be = ptr(a[9]), *ga = ptr(a[10]), *al = ptr(a[11]), *dt = ptr(a[12]), *no = ptr(a[13]);
    const float eps = f32(a[14]); void *S = ptr(a[15]), *out = ptr(a[16]);
    RUN(cwk_gdn_scan(c, B, n_, nh, hk, hv, grp, up, gd, be, ga, al, dt, no, eps, S, out));
})

static PyMethodDef methods[] = {
#define M(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, NULL}
    M(cwk_mla_decode), M(cwk_gqa_decode), M(cwk_dsa_select), M(cwk_gdn_scan), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__pycall(void) { return PyModule_Create(&module); }
