/* The hot entry points of libingot_qmm.so as CPython functions. A ctypes call converts every argument through its argtypes
 * object: 2.3 us for iq_qmv, half of what a decode linear of a few megabytes takes on the GPU; through METH_FASTCALL it is
 * 0.3 us. Arguments are integers (addresses, sizes, flags) and, where the C signature has them, floats; the result is the
 * status. The library is already loaded (capi.lib()); bind(name, address) hands over the symbols. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "../../include/ingot_qmm.h"

static void* fn_qmv;
static void* fn_qmm;
static void* fn_dense_ffn;
static void* fn_moe_forward;
static void* fn_rmsnorm;
static void* fn_had_rows;
static void* fn_embed_rows;
static void* fn_argmax_rows;
static void* fn_topk64;

static const struct { const char* name; void** slot; } table[] = {
    {"iq_qmv", &fn_qmv},           {"iq_qmm", &fn_qmm},               {"iq_dense_ffn", &fn_dense_ffn},
    {"iq_moe_forward", &fn_moe_forward}, {"iq_rmsnorm", &fn_rmsnorm}, {"iq_had_rows", &fn_had_rows},
    {"iq_embed_rows", &fn_embed_rows},   {"iq_argmax_rows", &fn_argmax_rows}, {"iq_topk64", &fn_topk64},
};

static PyObject* py_bind(PyObject* self, PyObject* args) {
    const char* name;
    unsigned long long addr;
    (void)self;
    if (!PyArg_ParseTuple(args, "sK", &name, &addr)) return NULL;
    for (size_t i = 0; i < sizeof(table) / sizeof(table[0]); i++)
        if (strcmp(table[i].name, name) == 0) {
            *table[i].slot = (void*)(uintptr_t)addr;
            Py_RETURN_NONE;
        }
    PyErr_Format(PyExc_KeyError, "no entry point %s", name);
    return NULL;
}

/* argument i as a 64-bit pattern; a conversion error is looked for once, after all of them */
static inline uint64_t U(PyObject* const* a, int i) {
    if (a[i] == Py_None) return 0;
    return PyLong_AsUnsignedLongLongMask(a[i]);
}
#define P(i) ((void*)(uintptr_t)U(a, i))
#define I32(i) ((int32_t)U(a, i))
#define I64(i) ((int64_t)U(a, i))
#define U32(i) ((uint32_t)U(a, i))
#define F32(i) ((float)PyFloat_AsDouble(a[i]))

#define ENTRY(NAME, COUNT, TYPE, ...)                                                                \
    static PyObject* py_##NAME(PyObject* self, PyObject* const* a, Py_ssize_t n) {                  \
        (void)self;                                                                                 \
        if (n != COUNT || fn_##NAME == NULL) {                                                      \
            PyErr_SetString(PyExc_TypeError, #NAME ": wrong number of arguments, or not bound");    \
            return NULL;                                                                            \
        }                                                                                           \
        TYPE f = (TYPE)fn_##NAME;                                                                   \
        int32_t st;                                                                                 \
        __VA_ARGS__;                                                                                 \
        return PyLong_FromLong(st);                                                                 \
    }
/* converts every argument first, so that nothing is launched when one of them is not a number */
#define CHECKED if (PyErr_Occurred()) return NULL
/* a launch can block on a full queue: other threads run meanwhile */
#define LAUNCH(CALL_) Py_BEGIN_ALLOW_THREADS st = CALL_; Py_END_ALLOW_THREADS

typedef int32_t (*qmv_t)(iq_ctx*, void*, const void*, int32_t, int64_t, const iq_qlinear*, void*, int32_t, int64_t, int32_t,
                         uint32_t, int32_t);
ENTRY(qmv, 12, qmv_t, {
    void *c = P(0), *s = P(1), *x = P(2), *q = P(5), *y = P(6);
    int32_t xd = I32(3), yd = I32(7), rows = I32(9), np = I32(11);
    int64_t ldx = I64(4), ldy = I64(8);
    uint32_t fl = U32(10);
    CHECKED;
    LAUNCH(f(c, s, x, xd, ldx, q, y, yd, ldy, rows, fl, np));
})
typedef int32_t (*qmm_t)(iq_ctx*, void*, const void*, int32_t, int64_t, const iq_qlinear*, void*, int32_t, int64_t, int32_t,
                         uint32_t, void*, size_t);
ENTRY(qmm, 13, qmm_t, {
    void *c = P(0), *s = P(1), *x = P(2), *q = P(5), *y = P(6), *ws = P(11);
    int32_t xd = I32(3), yd = I32(7), rows = I32(9);
    int64_t ldx = I64(4), ldy = I64(8);
    uint32_t fl = U32(10);
    size_t wb = (size_t)U(a, 12);
    CHECKED;
    LAUNCH(f(c, s, x, xd, ldx, q, y, yd, ldy, rows, fl, ws, wb));
})
typedef int32_t (*ffn_t)(iq_ctx*, void*, const void*, int32_t, int64_t, const iq_qlinear*, const iq_qlinear*, int32_t, float,
                         void*, int32_t, int64_t, int32_t, uint32_t, void*, size_t);
ENTRY(dense_ffn, 16, ffn_t, {
    void *c = P(0), *s = P(1), *x = P(2), *g = P(5), *d = P(6), *o = P(9), *ws = P(14);
    int32_t xd = I32(3), act = I32(7), od = I32(10), rows = I32(12);
    int64_t ldx = I64(4), ldo = I64(11);
    float lim = F32(8);
    uint32_t fl = U32(13);
    size_t wb = (size_t)U(a, 15);
    CHECKED;
    LAUNCH(f(c, s, x, xd, ldx, g, d, act, lim, o, od, ldo, rows, fl, ws, wb));
})
typedef int32_t (*moe_t)(iq_moe*, void*, const void*, int32_t, int64_t, void*, int32_t, int64_t, int32_t, uint32_t, uint32_t, void*,
                         size_t);
ENTRY(moe_forward, 13, moe_t, {
    void *l = P(0), *s = P(1), *x = P(2), *o = P(5), *ws = P(11);
    int32_t xd = I32(3), od = I32(6), rows = I32(8);
    int64_t ldx = I64(4), ldo = I64(7);
    uint32_t fl = U32(9), pieces = U32(10);
    size_t wb = (size_t)U(a, 12);
    CHECKED;
    LAUNCH(f(l, s, x, xd, ldx, o, od, ldo, rows, fl, pieces, ws, wb));
})
typedef int32_t (*norm_t)(iq_ctx*, void*, const float*, int64_t, void*, int32_t, int64_t, int32_t, int32_t, float);
ENTRY(rmsnorm, 10, norm_t, {
    void *c = P(0), *s = P(1), *x = P(2), *o = P(4);
    int64_t ldx = I64(3), ldo = I64(6);
    int32_t od = I32(5), rows = I32(7), d = I32(8);
    float eps = F32(9);
    CHECKED;
    LAUNCH(f(c, s, x, ldx, o, od, ldo, rows, d, eps));
})
typedef int32_t (*had_t)(iq_ctx*, void*, const void*, int32_t, int64_t, const float*, void*, int64_t, int32_t, int32_t);
ENTRY(had_rows, 10, had_t, {
    void *c = P(0), *s = P(1), *x = P(2), *sg = P(5), *y = P(6);
    int32_t xd = I32(3), rows = I32(8), k = I32(9);
    int64_t ldx = I64(4), ldy = I64(7);
    CHECKED;
    LAUNCH(f(c, s, x, xd, ldx, sg, y, ldy, rows, k));
})
typedef int32_t (*embed_t)(iq_ctx*, void*, const iq_qlinear*, const uint32_t*, int32_t, float*, void*, int64_t);
ENTRY(embed_rows, 8, embed_t, {
    void *c = P(0), *s = P(1), *q = P(2), *tok = P(3), *of = P(5), *oh = P(6);
    int32_t rows = I32(4);
    int64_t ldo = I64(7);
    CHECKED;
    LAUNCH(f(c, s, q, tok, rows, of, oh, ldo));
})
typedef int32_t (*argmax_t)(iq_ctx*, void*, const float*, int64_t, int32_t, int32_t, uint32_t*);
ENTRY(argmax_rows, 7, argmax_t, {
    void *c = P(0), *s = P(1), *x = P(2), *o = P(6);
    int64_t ldx = I64(3);
    int32_t rows = I32(4), nn = I32(5);
    CHECKED;
    LAUNCH(f(c, s, x, ldx, rows, nn, o));
})
typedef int32_t (*topk_t)(iq_ctx*, void*, const float*, int64_t, int32_t, int32_t, const float*, int32_t, uint32_t*, float*, float*,
                          void*, size_t);
ENTRY(topk64, 13, topk_t, {
    void *c = P(0), *s = P(1), *x = P(2), *t = P(6), *ix = P(8), *v = P(9), *z = P(10), *sc = P(11);
    int64_t ldx = I64(3);
    int32_t rows = I32(4), vocab = I32(5), nt = I32(7);
    size_t sb = (size_t)U(a, 12);
    CHECKED;
    LAUNCH(f(c, s, x, ldx, rows, vocab, t, nt, ix, v, z, sc, sb));
})

#define M(NAME) {#NAME, (PyCFunction)(void (*)(void))py_##NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, NULL}, M(qmv), M(qmm), M(dense_ffn), M(moe_forward), M(rmsnorm), M(had_rows), M(embed_rows),
    M(argmax_rows), M(topk64), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_iqcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__iqcall(void) { return PyModule_Create(&module); }
