/* The operator calls of the Python binding without ctypes: arguments go from the binding's objects straight into the
 * C ABI's structs. A GEMV's ctypes call took 2.9 us of 5.1 for its conversions (5.7 us for the nine structs of q/k/v);
 * here they take 0.5. Each function returns True when the operator was called and succeeded, raises the binding's error when it
 * was refused, and returns False, with nothing called, when an argument is not what it knows how to read: the caller then goes
 * through ctypes, which converts or rejects it as before. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/tessl_b200.h"

static PyObject *s_handle, *s_value, *s_ptr, *s_nbytes, *s_packed, *s_sb, *s_rows, *s_cols, *s_group, *s_q, *s_k, *s_v;
static PyObject *error_class; /* TesslError(status, message) */

/* Readers: 1 if the object was understood. An int is taken modulo 2^32 or 2^64, as a ctypes integer argument is. */
static int as_u64(PyObject *o, uint64_t *out)
{
    if (!PyLong_Check(o)) return 0;
    *out = PyLong_AsUnsignedLongLongMask(o);
    return 1;
}
static int as_u32(PyObject *o, uint32_t *out)
{
    uint64_t v;
    if (!as_u64(o, &v)) return 0;
    *out = (uint32_t)v;
    return 1;
}
static int attr_u64(PyObject *o, PyObject *name, uint64_t *out)
{
    PyObject *v = PyObject_GetAttr(o, name);
    if (!v) return 0;
    const int ok = as_u64(v, out);
    Py_DECREF(v);
    return ok;
}
static int attr_u32(PyObject *o, PyObject *name, uint32_t *out)
{
    uint64_t v;
    if (!attr_u64(o, name, &v)) return 0;
    *out = (uint32_t)v;
    return 1;
}
static int as_flag(PyObject *o, uint32_t *out)
{
    *out = o == Py_True;
    return PyBool_Check(o);
}
static int as_f32(PyObject *o, float *out)
{
    if (!PyFloat_Check(o)) return 0;
    *out = (float)PyFloat_AS_DOUBLE(o);
    return 1;
}
static int as_buf(PyObject *o, TesslBuf *out)
{
    uint64_t p, n;
    if (!attr_u64(o, s_ptr, &p) || !attr_u64(o, s_nbytes, &n)) return 0;
    out->ptr = (void *)(uintptr_t)p;
    out->nbytes = n;
    return 1;
}
static int attr_buf(PyObject *o, PyObject *name, TesslBuf *out)
{
    PyObject *v = PyObject_GetAttr(o, name);
    if (!v) return 0;
    const int ok = as_buf(v, out);
    Py_DECREF(v);
    return ok;
}
static int as_bank(PyObject *o, TesslQ4MlxBank *out)
{
    return attr_buf(o, s_packed, &out->packed) && attr_buf(o, s_sb, &out->scales_biases);
}
static int as_qkv(PyObject *o, TesslQkvOutputs *out)
{
    return attr_buf(o, s_q, &out->q_out) && attr_buf(o, s_k, &out->k_out) && attr_buf(o, s_v, &out->v_out);
}
static int as_shape(PyObject *o, TesslQuantShape *out)
{
    return attr_u32(o, s_rows, &out->rows) && attr_u32(o, s_cols, &out->cols) && attr_u32(o, s_group, &out->group_size);
}
/* An optional buffer: *out points to *store, or is NULL for None. */
static int as_opt(PyObject *o, TesslBuf *store, const TesslBuf **out)
{
    *out = NULL;
    if (o == Py_None) return 1;
    *out = store;
    return as_buf(o, store);
}
/* The runtime's handle, a c_void_p (None once it is closed). */
static int as_rt(PyObject *o, TesslRuntime **out)
{
    PyObject *h = PyObject_GetAttr(o, s_handle);
    if (!h) return 0;
    PyObject *v = h == Py_None ? Py_NewRef(Py_None) : PyObject_GetAttr(h, s_value);
    Py_DECREF(h);
    if (!v) return 0;
    uint64_t p = 0;
    const int ok = v == Py_None || as_u64(v, &p);
    Py_DECREF(v);
    *out = (TesslRuntime *)(uintptr_t)p;
    return ok;
}

static PyObject *not_understood(void)
{
    PyErr_Clear();
    Py_RETURN_FALSE;
}
static PyObject *finish(int32_t status, const char *err)
{
    if (status == TESSL_OK) Py_RETURN_TRUE;
    PyObject *msg = PyUnicode_DecodeUTF8(err, (Py_ssize_t)strlen(err), "replace");
    if (!msg) return NULL;
    PyObject *e = PyObject_CallFunction(error_class, "iO", (int)status, msg);
    Py_DECREF(msg);
    if (e) {
        PyErr_SetObject(error_class, e);
        Py_DECREF(e);
    }
    return NULL;
}

/* The call itself, without the interpreter lock (a synchronous runtime waits for the GPU in it). */
#define RUN(expr)                                        \
    do {                                                 \
        char err[1024];                                  \
        int32_t status;                                  \
        err[0] = 0;                                      \
        Py_BEGIN_ALLOW_THREADS status = (expr);          \
        Py_END_ALLOW_THREADS return finish(status, err); \
    } while (0)
#define OP(name) static PyObject *op_##name(PyObject *self, PyObject *const *a, Py_ssize_t n)
#define NEED(count, cond) \
    if (n != (count) || !(cond)) return not_understood()

OP(gemv_q4_mlx_simd) /* rt, bank, x, y, shape, layout, resid, bf16 */
{
    TesslRuntime *rt;
    TesslQ4MlxBank b;
    TesslBuf x, y, rs;
    TesslQuantShape s;
    uint32_t layout, bf16;
    const TesslBuf *r;
    NEED(8, as_rt(a[0], &rt) && as_bank(a[1], &b) && as_buf(a[2], &x) && as_buf(a[3], &y) && as_shape(a[4], &s) &&
                as_u32(a[5], &layout) && as_opt(a[6], &rs, &r) && as_flag(a[7], &bf16));
    if (bf16) RUN(tessl_gemv_q4_mlx_simd_bf16(rt, b, x, y, s, layout, r, err, sizeof err));
    RUN(tessl_gemv_q4_mlx_simd(rt, b, x, y, s, layout, r, err, sizeof err));
}
OP(gemv_q4_mlx_gate_up_silu) /* rt, gate, up, x, mid, shape, bf16 */
{
    TesslRuntime *rt;
    TesslQ4MlxBank g, u;
    TesslBuf x, mid;
    TesslQuantShape s;
    uint32_t bf16;
    NEED(7, as_rt(a[0], &rt) && as_bank(a[1], &g) && as_bank(a[2], &u) && as_buf(a[3], &x) && as_buf(a[4], &mid) &&
                as_shape(a[5], &s) && as_flag(a[6], &bf16));
    RUN(tessl_gemv_q4_mlx_gate_up_silu(rt, g, u, x, mid, s, bf16, err, sizeof err));
}
OP(gemv_q4_mlx_kv) /* rt, k, v, x, k_out, v_out, shape, layout */
{
    TesslRuntime *rt;
    TesslQ4MlxBank k, v;
    TesslBuf x, ko, vo;
    TesslQuantShape s;
    uint32_t layout;
    NEED(8, as_rt(a[0], &rt) && as_bank(a[1], &k) && as_bank(a[2], &v) && as_buf(a[3], &x) && as_buf(a[4], &ko) &&
                as_buf(a[5], &vo) && as_shape(a[6], &s) && as_u32(a[7], &layout));
    RUN(tessl_gemv_q4_mlx_kv(rt, k, v, x, ko, vo, s, layout, err, sizeof err));
}
OP(gemv_q4_mlx_qkv) /* rt, q, k, v, x, out, rows_q, rows_kv, cols, group, layout */
{
    TesslRuntime *rt;
    TesslQ4MlxBank q, k, v;
    TesslBuf x;
    TesslQkvOutputs out;
    uint32_t rq, rkv, cols, group, layout;
    NEED(11, as_rt(a[0], &rt) && as_bank(a[1], &q) && as_bank(a[2], &k) && as_bank(a[3], &v) && as_buf(a[4], &x) &&
                 as_qkv(a[5], &out) && as_u32(a[6], &rq) && as_u32(a[7], &rkv) && as_u32(a[8], &cols) && as_u32(a[9], &group) &&
                 as_u32(a[10], &layout));
    RUN(tessl_gemv_q4_mlx_qkv(rt, q, k, v, x, out, rq, rkv, cols, group, layout, err, sizeof err));
}
OP(swiglu) /* rt, gate, up, out, n, bf16 */
{
    TesslRuntime *rt;
    TesslBuf g, u, o;
    uint32_t count, bf16;
    NEED(6, as_rt(a[0], &rt) && as_buf(a[1], &g) && as_buf(a[2], &u) && as_buf(a[3], &o) && as_u32(a[4], &count) &&
                as_flag(a[5], &bf16));
    RUN(tessl_swiglu(rt, g, u, o, count, bf16, err, sizeof err));
}
OP(gemm_q4_mlx) /* rt, bank, x, y, shape, m, layout, resid, bf16 */
{
    TesslRuntime *rt;
    TesslQ4MlxBank b;
    TesslBuf x, y, rs;
    TesslQuantShape s;
    uint32_t m, layout, bf16;
    const TesslBuf *r;
    NEED(9, as_rt(a[0], &rt) && as_bank(a[1], &b) && as_buf(a[2], &x) && as_buf(a[3], &y) && as_shape(a[4], &s) && as_u32(a[5], &m) &&
                as_u32(a[6], &layout) && as_opt(a[7], &rs, &r) && as_flag(a[8], &bf16));
    if (bf16) RUN(tessl_gemm_q4_mlx_bf16(rt, b, x, y, s, m, layout, r, err, sizeof err));
    RUN(tessl_gemm_q4_mlx(rt, b, x, y, s, m, layout, r, err, sizeof err));
}
OP(gemm_q4_mlx_tensorops) /* rt, bank, x, y, shape, m, bf16 */
{
    TesslRuntime *rt;
    TesslQ4MlxBank b;
    TesslBuf x, y;
    TesslQuantShape s;
    uint32_t m, bf16;
    NEED(7, as_rt(a[0], &rt) && as_bank(a[1], &b) && as_buf(a[2], &x) && as_buf(a[3], &y) && as_shape(a[4], &s) && as_u32(a[5], &m) &&
                as_flag(a[6], &bf16));
    if (bf16) RUN(tessl_gemm_q4_mlx_tensorops_bf16(rt, b, x, y, s, m, err, sizeof err));
    RUN(tessl_gemm_q4_mlx_tensorops(rt, b, x, y, s, m, err, sizeof err));
}
OP(gemv_q8) /* rt, packed, scales, zeros, x, y, rows, cols, group */
{
    TesslRuntime *rt;
    TesslBuf q, sc, z, x, y;
    uint32_t rows, cols, group;
    NEED(9, as_rt(a[0], &rt) && as_buf(a[1], &q) && as_buf(a[2], &sc) && as_buf(a[3], &z) && as_buf(a[4], &x) && as_buf(a[5], &y) &&
                as_u32(a[6], &rows) && as_u32(a[7], &cols) && as_u32(a[8], &group));
    RUN(tessl_gemv_q8(rt, q, sc, z, x, y, rows, cols, group, err, sizeof err));
}
OP(gemm_q8_mlx) /* rt, codes, sb, x, y, shape, m, bf16 */
{
    TesslRuntime *rt;
    TesslBuf q, sb, x, y;
    TesslQuantShape s;
    uint32_t m, bf16;
    NEED(8, as_rt(a[0], &rt) && as_buf(a[1], &q) && as_buf(a[2], &sb) && as_buf(a[3], &x) && as_buf(a[4], &y) && as_shape(a[5], &s) &&
                as_u32(a[6], &m) && as_flag(a[7], &bf16));
    RUN(tessl_gemm_q8_mlx(rt, q, sb, x, y, s, m, bf16, err, sizeof err));
}
OP(embed_lookup_q4_mlx) /* rt, bank, ids, out, vocab, hidden, group, tokens */
{
    TesslRuntime *rt;
    TesslQ4MlxBank b;
    TesslBuf ids, out;
    uint32_t vocab, hidden, group, tokens;
    NEED(8, as_rt(a[0], &rt) && as_bank(a[1], &b) && as_buf(a[2], &ids) && as_buf(a[3], &out) && as_u32(a[4], &vocab) &&
                as_u32(a[5], &hidden) && as_u32(a[6], &group) && as_u32(a[7], &tokens));
    RUN(tessl_embed_lookup_q4_mlx(rt, b, ids, out, vocab, hidden, group, tokens, err, sizeof err));
}
OP(qwen35_rms_norm) /* rt, x, w, out, bf16, rows, dim, eps */
{
    TesslRuntime *rt;
    TesslBuf x, w, o;
    uint32_t bf16, rows, dim;
    float eps;
    NEED(8, as_rt(a[0], &rt) && as_buf(a[1], &x) && as_buf(a[2], &w) && as_buf(a[3], &o) && as_flag(a[4], &bf16) &&
                as_u32(a[5], &rows) && as_u32(a[6], &dim) && as_f32(a[7], &eps));
    RUN(tessl_qwen35_rms_norm(rt, x, w, o, bf16, rows, dim, eps, err, sizeof err));
}
OP(qwen35_residual_add) /* rt, y, resid, rows, width */
{
    TesslRuntime *rt;
    TesslBuf y, r;
    uint32_t rows, width;
    NEED(5, as_rt(a[0], &rt) && as_buf(a[1], &y) && as_buf(a[2], &r) && as_u32(a[3], &rows) && as_u32(a[4], &width));
    RUN(tessl_qwen35_residual_add(rt, y, r, rows, width, err, sizeof err));
}
OP(qwen35_add_rms_norm) /* rt, y, resid, w, out, bf16, rows, dim, eps */
{
    TesslRuntime *rt;
    TesslBuf y, r, w, o;
    uint32_t bf16, rows, dim;
    float eps;
    NEED(9, as_rt(a[0], &rt) && as_buf(a[1], &y) && as_buf(a[2], &r) && as_buf(a[3], &w) && as_buf(a[4], &o) && as_flag(a[5], &bf16) &&
                as_u32(a[6], &rows) && as_u32(a[7], &dim) && as_f32(a[8], &eps));
    RUN(tessl_qwen35_add_rms_norm(rt, y, r, w, o, bf16, rows, dim, eps, err, sizeof err));
}

static PyObject *set_error(PyObject *self, PyObject *cls)
{
    Py_XSETREF(error_class, Py_NewRef(cls));
    Py_RETURN_NONE;
}

#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))op_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    ENTRY(gemv_q4_mlx_simd), ENTRY(gemv_q4_mlx_gate_up_silu), ENTRY(gemv_q4_mlx_kv), ENTRY(gemv_q4_mlx_qkv), ENTRY(swiglu),
    ENTRY(gemm_q4_mlx), ENTRY(gemm_q4_mlx_tensorops), ENTRY(gemv_q8), ENTRY(gemm_q8_mlx), ENTRY(embed_lookup_q4_mlx),
    ENTRY(qwen35_rms_norm), ENTRY(qwen35_residual_add), ENTRY(qwen35_add_rms_norm),
    {"set_error", set_error, METH_O, "The class to raise refusals as: called with (status, message)."},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tessl_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__tessl_call(void)
{
    struct {
        PyObject **at;
        const char *name;
    } names[] = {{&s_handle, "handle"}, {&s_value, "value"}, {&s_ptr, "ptr"}, {&s_nbytes, "nbytes"}, {&s_packed, "packed"},
                 {&s_sb, "scales_biases"}, {&s_rows, "rows"}, {&s_cols, "cols"}, {&s_group, "group_size"}, {&s_q, "q_out"},
                 {&s_k, "k_out"}, {&s_v, "v_out"}};
    for (size_t i = 0; i < sizeof names / sizeof names[0]; ++i)
        if (!(*names[i].at = PyUnicode_InternFromString(names[i].name))) return NULL;
    error_class = Py_NewRef(PyExc_RuntimeError);
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddIntConstant(m, "ABI_VERSION", TESSL_B200_ABI_VERSION) < 0) Py_CLEAR(m);
    return m;
}
