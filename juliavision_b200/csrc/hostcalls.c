// The host side of the entry points that a program calls many times a second, as a CPython extension: the checks of
// the operands and the call into libb200dnn in one step.  What bounds a call on a few hundred tokens is not the GPU but
// the interpreter: the same checks and a ctypes call of 17 arguments in Python took 11 us for matmul_ and 13 us for
// sdpa before the library was entered, against 4 to 8 us of device time; here they take 0.7.  A call of 363 tokens
// through a 240 x 1496 projection went from 11.6 to 4.9 us, an attention of 42 x 3 windows of 196 from 13.0 to 7.9.
//
// Each function takes the forms a program ordinarily passes and answers None for every other one, which the Python
// route then takes, declines or refuses exactly as it always has; nothing is decided here that it would decide
// differently.  The library is entered without the interpreter's lock, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "../../include/b200dnn.h"

typedef struct {
    int64_t ptr, shape[4], stride[4], size;
    int nd, code;
} Arr;

static PyObject *s_ptr, *s_dtype, *s_shape, *s_strides;
static PyObject *dt_f16, *dt_f32;   // numpy's own dtype objects; an equal one that is not the same goes the Python route

static int (*p_gemm)(b200_ctx*, int64_t, int64_t, int64_t, const void*, int64_t, const void*, int64_t, const void*, void*,
                     int64_t, int, int, int64_t, int64_t, int64_t, int64_t);
static int (*p_gemv)(b200_ctx*, int64_t, int64_t, const void*, int64_t, const void*, const void*, int, void*, int, int);
static int (*p_attention)(b200_ctx*, int64_t, int64_t, int64_t, int64_t, int64_t, const b200_strided4*, const b200_strided4*,
                          const b200_strided4*, const b200_strided4*, const b200_strided4*, int, float);
static int (*p_layernorm)(b200_ctx*, int64_t, int64_t, const void*, int, void*, int, float*, float*, const void*, const void*,
                          float);
static int (*p_conv)(b200_ctx*, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                     int64_t, int64_t, int64_t, const void*, const void*, const void*, void*, int, int);

static int64_t attr_int(PyObject* o, PyObject* name, int* ok) {
    PyObject* v = PyObject_GetAttr(o, name);
    int64_t r = 0;
    if (v && PyLong_Check(v)) r = PyLong_AsLongLong(v);
    else *ok = 0;
    Py_XDECREF(v);
    return r;
}

static int ints(PyObject* t, int64_t* out, int n) {   // a tuple of n integers
    if (!t || !PyTuple_Check(t) || PyTuple_GET_SIZE(t) != n) return 0;
    for (int i = 0; i < n; ++i) {
        PyObject* v = PyTuple_GET_ITEM(t, i);
        if (!PyLong_Check(v)) return 0;
        out[i] = PyLong_AsLongLong(v);
    }
    return !PyErr_Occurred();
}

// A DeviceArray of fp16 or fp32 with one to four axes and a size that is a number here; 0 for anything else.
static int load(PyObject* o, Arr* a) {
    int ok;
    PyObject* dt = PyObject_GetAttr(o, s_dtype);
    a->code = dt == dt_f16 ? B200_F16 : dt == dt_f32 ? B200_F32 : -1;
    Py_XDECREF(dt);   // numpy holds the two that count
    ok = a->code >= 0;
    a->ptr = ok ? attr_int(o, s_ptr, &ok) : 0;
    if (ok) {
        PyObject *sh = PyObject_GetAttr(o, s_shape), *st = PyObject_GetAttr(o, s_strides);
        a->nd = sh && PyTuple_Check(sh) ? (int)PyTuple_GET_SIZE(sh) : 0;
        ok = a->nd >= 1 && a->nd <= 4 && ints(sh, a->shape, a->nd) && ints(st, a->stride, a->nd);
        a->size = 1;
        for (int i = 0; ok && i < a->nd; ++i) ok = a->shape[i] >= 0 && !__builtin_mul_overflow(a->size, a->shape[i], &a->size);
        Py_XDECREF(sh);
        Py_XDECREF(st);
    }
    if (PyErr_Occurred()) {   // an attribute that is missing or out of range: the Python route meets it again
        PyErr_Clear();
        ok = 0;
    }
    return ok;
}

static int dense(const Arr* a) {
    int64_t acc = 1;
    for (int i = 0; i < a->nd; ++i) {
        if (a->shape[i] != 1 && a->stride[i] != acc) return 0;
        acc *= a->shape[i];
    }
    return 1;
}
static int64_t colmajor(const Arr* a) {   // leading dimension of a 2-D view with a unit first stride, else -1
    if (a->shape[0] != 1 && a->stride[0] != 1) return -1;
    const int64_t ld = a->shape[1] != 1 ? a->stride[1] : (a->shape[0] > 1 ? a->shape[0] : 1);
    return ld >= a->shape[0] ? ld : -1;
}
// A dense vector of n elements of one type, or None: 1 with *p set, else 0.
static int vector(PyObject* o, int code, int64_t n, const void** p) {
    Arr a;
    *p = NULL;
    if (o == Py_None) return 1;
    if (!load(o, &a) || a.code != code || a.size != n || !dense(&a)) return 0;
    *p = (const void*)a.ptr;
    return 1;
}

#define P(a) ((void*)(a).ptr)
#define ENTER(rc, call)          \
    do {                         \
        Py_BEGIN_ALLOW_THREADS   \
        rc = (call);             \
        Py_END_ALLOW_THREADS     \
    } while (0)

static b200_ctx* handle(PyObject* o) {
    if (!PyLong_Check(o)) return NULL;
    void* p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) PyErr_Clear();
    return (b200_ctx*)p;
}
static int epilogue(PyObject* o) { return PyLong_Check(o) ? (int)PyLong_AsLong(o) : -1; }

// matmul(handle, out, A, B, bias, epilogue)
static PyObject* h_matmul(PyObject* self, PyObject* const* v, Py_ssize_t n) {
    Arr out, A, B;
    const void* bias;
    b200_ctx* c;
    int epi, rc;
    if (n != 6 || !(c = handle(v[0])) || (epi = epilogue(v[5])) < 0) Py_RETURN_NONE;
    if (!load(v[1], &out) || !load(v[2], &A) || !load(v[3], &B) || out.nd != 2 || A.nd != 2 || B.nd != 2) Py_RETURN_NONE;
    const int64_t M = A.shape[0], K = A.shape[1], N = B.shape[1], lim = (int64_t)1 << 31;
    const int64_t lda = colmajor(&A), ldb = colmajor(&B), ldo = colmajor(&out);
    if (A.code != B.code || B.shape[0] != K || out.shape[0] != M || out.shape[1] != N || lda < 0 || ldb < 0 || ldo < 0 ||
        M < 1 || N < 1 || K < 1 || M >= lim || N >= lim || K >= lim || !vector(v[4], A.code, M, &bias))
        Py_RETURN_NONE;
    if (N == 1) {
        if (!dense(&B) || !dense(&out) || (out.code != B200_F32 && out.code != A.code)) Py_RETURN_NONE;
        ENTER(rc, p_gemv(c, M, K, P(A), lda, P(B), bias, A.code, P(out), out.code, epi));
    } else {
        if (A.code != B200_F16) Py_RETURN_NONE;
        ENTER(rc, p_gemm(c, M, N, K, P(A), lda, P(B), ldb, bias, P(out), ldo, out.code, epi, 1, 0, 0, 0));
    }
    return PyLong_FromLong(rc);
}

static void strided(const Arr* a, b200_strided4* s) {
    s->ptr = (const void*)a->ptr;
    for (int i = 0; i < 4; ++i) s->stride[i] = a->stride[i];
}

// sdpa(handle, out, q, k, v, bias, scale)
static PyObject* h_sdpa(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    Arr out, q, k, v, b;
    b200_ctx* c;
    int rc;
    if (n != 7 || !(c = handle(a[0])) || !PyFloat_Check(a[6])) Py_RETURN_NONE;
    if (!load(a[1], &out) || !load(a[2], &q) || !load(a[3], &k) || !load(a[4], &v)) Py_RETURN_NONE;
    if (out.nd != 4 || q.nd != 4 || k.nd != 4 || v.nd != 4 || q.code != B200_F16 || k.code != B200_F16 || v.code != B200_F16)
        Py_RETURN_NONE;
    const int64_t E = q.shape[0], Lq = q.shape[1], H = q.shape[2], B = q.shape[3], Lk = k.shape[1], lim = (int64_t)1 << 31;
    if (E < 8 || E > 128 || E % 8 || Lq < 1 || Lk < 1 || Lq >= lim || Lk >= lim || H < 1 || H > 65535 || B < 1 || B > 65535)
        Py_RETURN_NONE;
    for (int i = 0; i < 4; ++i)
        if (k.shape[i] != (i == 1 ? Lk : q.shape[i]) || v.shape[i] != k.shape[i] || out.shape[i] != q.shape[i]) Py_RETURN_NONE;
    if (q.stride[0] != 1 || k.stride[0] != 1 || v.stride[0] != 1 || out.stride[0] != 1) Py_RETURN_NONE;
    b200_strided4 sq, sk, sv, so, sb;
    strided(&q, &sq);
    strided(&k, &sk);
    strided(&v, &sv);
    strided(&out, &so);
    const int masked = a[5] != Py_None;
    if (masked) {
        const int64_t want[4] = {Lk, Lq, H, B};
        if (!load(a[5], &b) || b.nd != 4 || b.code != B200_F16) Py_RETURN_NONE;
        for (int i = 0; i < 4; ++i) {
            if (b.shape[i] != 1 && b.shape[i] != want[i]) Py_RETURN_NONE;
            if (b.shape[i] == 1) b.stride[i] = 0;   // a size-1 axis broadcasts
        }
        strided(&b, &sb);
    }
    const float scale = (float)PyFloat_AS_DOUBLE(a[6]);
    ENTER(rc, p_attention(c, E, Lq, Lk, H, B, &sq, &sk, &sv, masked ? &sb : NULL, &so, out.code, scale));
    return PyLong_FromLong(rc);
}

// layernorm(handle, out, mean, rstd, a, gamma, beta, C, eps)
static PyObject* h_layernorm(PyObject* self, PyObject* const* v, Py_ssize_t n) {
    Arr out, mean, rstd, a;
    const void *gamma, *beta;
    b200_ctx* c;
    int rc;
    if (n != 9 || !(c = handle(v[0])) || !PyLong_Check(v[7]) || !PyFloat_Check(v[8])) Py_RETURN_NONE;
    if (!load(v[1], &out) || !load(v[2], &mean) || !load(v[3], &rstd) || !load(v[4], &a)) Py_RETURN_NONE;
    int over;
    const int64_t C = PyLong_AsLongLongAndOverflow(v[7], &over), total = a.size;
    if (over || C < 1 || total % C || out.size != total || !dense(&a) || !dense(&out) || !dense(&mean) || !dense(&rstd)) Py_RETURN_NONE;
    const int64_t groups = total / C;
    if (mean.code != B200_F32 || rstd.code != B200_F32 || mean.size < groups || rstd.size < groups) Py_RETURN_NONE;
    if (!vector(v[5], a.code, C, &gamma) || !vector(v[6], a.code, C, &beta)) Py_RETURN_NONE;
    const float eps = (float)PyFloat_AS_DOUBLE(v[8]);
    ENTER(rc, p_layernorm(c, groups, C, P(a), a.code, P(out), out.code, (float*)P(mean), (float*)P(rstd), gamma, beta, eps));
    return PyLong_FromLong(rc);
}

// convolution(handle, out, x, w, bias, stride, padding, dilation, groups, act)
static PyObject* h_convolution(PyObject* self, PyObject* const* v, Py_ssize_t n) {
    Arr out, x, w;
    int64_t s[2], p[2], d[2];
    b200_ctx* c;
    int act, rc, over;
    if (n != 10 || !(c = handle(v[0])) || !PyLong_Check(v[8]) || (act = epilogue(v[9])) < 0) Py_RETURN_NONE;
    const int64_t groups = PyLong_AsLongLongAndOverflow(v[8], &over);
    if (over || !ints(v[5], s, 2) || !ints(v[6], p, 2) || !ints(v[7], d, 2)) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    if (!load(v[1], &out) || !load(v[2], &x) || !load(v[3], &w) || out.nd != 4 || x.nd != 4 || w.nd != 4) Py_RETURN_NONE;
    if (x.code != B200_F16 || w.code != B200_F16 || !dense(&x) || !dense(&w) || !dense(&out)) Py_RETURN_NONE;
    const void* bias;
    if (!vector(v[4], B200_F16, w.shape[3], &bias)) Py_RETURN_NONE;
    if (groups < 1 || w.shape[2] * groups != x.shape[2] || w.shape[3] % groups || out.shape[2] != w.shape[3] || out.shape[3] != x.shape[3])
        Py_RETURN_NONE;
    const int64_t lim = (int64_t)1 << 31;   // past it (no extent of a real convolution) the sums below could wrap
    for (int i = 0; i < 2; ++i) {
        if (x.shape[i] >= lim || w.shape[i] >= lim || s[i] >= lim || p[i] >= lim || d[i] >= lim) Py_RETURN_NONE;
        const int64_t span = x.shape[i] + 2 * p[i] - d[i] * (w.shape[i] - 1) - 1;
        if (s[i] < 1 || d[i] < 1 || p[i] < 0 || span < 0 || out.shape[i] != span / s[i] + 1) Py_RETURN_NONE;
    }
    ENTER(rc, p_conv(c, x.shape[0], x.shape[1], x.shape[2], x.shape[3], w.shape[0], w.shape[1], w.shape[3], s[0], s[1], p[0], p[1],
                     d[0], d[1], groups, P(x), P(w), bias, P(out), out.code, act));
    return PyLong_FromLong(rc);
}

// bind(gemm, gemv, attention, layernorm, convolution): the library's entry points, as addresses
static PyObject* h_bind(PyObject* self, PyObject* args) {
    unsigned long long a, b, c, d, e;
    if (!PyArg_ParseTuple(args, "KKKKK", &a, &b, &c, &d, &e)) return NULL;
    *(void**)&p_gemm = (void*)(uintptr_t)a;
    *(void**)&p_gemv = (void*)(uintptr_t)b;
    *(void**)&p_attention = (void*)(uintptr_t)c;
    *(void**)&p_layernorm = (void*)(uintptr_t)d;
    *(void**)&p_conv = (void*)(uintptr_t)e;
    Py_RETURN_NONE;
}

static PyMethodDef methods[] = {{"bind", h_bind, METH_VARARGS, NULL},
                                {"matmul", (PyCFunction)(void (*)(void))h_matmul, METH_FASTCALL, NULL},
                                {"sdpa", (PyCFunction)(void (*)(void))h_sdpa, METH_FASTCALL, NULL},
                                {"layernorm", (PyCFunction)(void (*)(void))h_layernorm, METH_FASTCALL, NULL},
                                {"convolution", (PyCFunction)(void (*)(void))h_convolution, METH_FASTCALL, NULL},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "hostcalls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_hostcalls(void) {
    s_ptr = PyUnicode_InternFromString("ptr");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_shape = PyUnicode_InternFromString("shape");
    s_strides = PyUnicode_InternFromString("strides");
    if (!s_ptr || !s_dtype || !s_shape || !s_strides) return NULL;
    PyObject* np = PyImport_ImportModule("numpy");
    if (!np) return NULL;
    dt_f16 = PyObject_CallMethod(np, "dtype", "s", "float16");
    dt_f32 = PyObject_CallMethod(np, "dtype", "s", "float32");
    Py_DECREF(np);
    if (!dt_f16 || !dt_f32) return NULL;
    return PyModule_Create(&module);
}
