/* Host path of the per-op calls of the Python mirror (ops.py): argument checks, the current stream and the library call in one C
 * function per op.  The same in Python and ctypes took 4 to 5 us of the 8 us between two calls of a small product, more than the
 * kernel; the checks, their order and their errors are those of the Python code before it.
 *
 * setup() hands over the classes, torch's two stream functions and the addresses of the library's entry points. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

static PyObject *s_is_cuda, *s_dtype, *s_is_contiguous, *s_data_ptr, *s_numel, *s_shape, *s_h, *s_value, *s_nrows, *s_ncols;
static PyObject *tensor_type, *float32, *get_device, *raw_stream, *wgb_error, *check_status, *rope_config, *attn_params;

enum { F_GEMV, F_GEMM_Q4K, F_GEMM_Q6K, F_GEMM_Q80, F_RMS_NORM, F_ROPE, F_ATTENTION, F_SILU, F_OP_ASSIGN, F_COUNT };
static void *fn[F_COUNT];
static const char *const entry[F_COUNT] = {   /* ENTRY_POINTS of the module: whose addresses setup() wants, in this order */
    "wgb_gemv_quant", "wgb_gemm_q4k_tiles", "wgb_gemm_q6k_tiles", "wgb_gemm_q80_tiles", "wgb_rms_norm", "wgb_rope", "wgb_attention", "wgb_silu", "wgb_op_assign",
};

static const long ERR_INVALID = 1;

static PyObject *setup(PyObject *self, PyObject *args)
{
    PyObject *addresses;
    if (!PyArg_ParseTuple(args, "OOOOOOOOO!", &tensor_type, &float32, &get_device, &raw_stream, &wgb_error, &check_status, &rope_config, &attn_params,
                          &PyTuple_Type, &addresses))
        return NULL;
    if (PyTuple_GET_SIZE(addresses) != F_COUNT) return PyErr_Format(PyExc_ValueError, "expected %d addresses", (int)F_COUNT);
    for (int i = 0; i < F_COUNT; i++) {
        fn[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(addresses, i));
        if (!fn[i]) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "null address");
    }
    PyObject *keep[] = { tensor_type, float32, get_device, raw_stream, wgb_error, check_status, rope_config, attn_params };
    for (size_t i = 0; i < sizeof(keep) / sizeof(keep[0]); i++) Py_INCREF(keep[i]);
    Py_RETURN_NONE;
}

static int expect(Py_ssize_t n, Py_ssize_t want)
{
    if (n == want && fn[0]) return 1;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments after setup()", want);
    return 0;
}

static PyObject *invalid(const char *message)
{
    PyObject *e = PyObject_CallFunction(wgb_error, "ls", ERR_INVALID, message);
    if (e) {
        PyErr_SetObject(wgb_error, e);
        Py_DECREF(e);
    }
    return NULL;
}

/* The value of a status: None, or what check() raises. */
static PyObject *finish(int status)
{
    if (status == 0) Py_RETURN_NONE;
    return PyObject_CallFunction(check_status, "i", status);
}

static int as_size(PyObject *o, size_t *out)   /* steals the reference */
{
    if (!o) return 0;
    *out = PyLong_AsSize_t(o);
    Py_DECREF(o);
    return !(*out == (size_t)-1 && PyErr_Occurred());
}
static int numel(PyObject *t, size_t *out) { return as_size(PyObject_CallMethodNoArgs(t, s_numel), out); }
static int attr_size(PyObject *o, PyObject *name, size_t *out) { return as_size(PyObject_GetAttr(o, name), out); }

static int truth(PyObject *o)   /* steals the reference; -1: error */
{
    if (!o) return -1;
    const int r = PyObject_IsTrue(o);
    Py_DECREF(o);
    return r;
}

/* Address of a contiguous float32 CUDA tensor. */
static int f32(PyObject *t, const char *name, void **out)
{
    int ok = (PyObject *)Py_TYPE(t) == tensor_type ? 1 : PyObject_IsInstance(t, tensor_type);
    if (ok > 0) ok = truth(PyObject_GetAttr(t, s_is_cuda));
    if (ok > 0) {
        PyObject *d = PyObject_GetAttr(t, s_dtype);
        if (!d) return 0;
        ok = d == float32;
        Py_DECREF(d);
    }
    if (ok > 0) ok = truth(PyObject_CallMethodNoArgs(t, s_is_contiguous));
    if (ok < 0) return 0;
    if (!ok) {
        PyErr_Format(PyExc_TypeError, "%s: expected a contiguous float32 CUDA tensor", name);
        return 0;
    }
    PyObject *p = PyObject_CallMethodNoArgs(t, s_data_ptr);
    if (!p) return 0;
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return *out || !PyErr_Occurred();
}

static int current_stream(void **out)
{
    PyObject *d = PyObject_CallNoArgs(get_device);
    if (!d) return 0;
    PyObject *s = PyObject_CallOneArg(raw_stream, d);
    Py_DECREF(d);
    if (!s) return 0;
    *out = PyLong_AsVoidPtr(s);
    Py_DECREF(s);
    return *out || !PyErr_Occurred();
}

/* The library's object behind a Python one (its ctypes handle `_h`; None once destroyed: the library's error follows). */
static int handle(PyObject *o, void **out)
{
    PyObject *h = PyObject_GetAttr(o, s_h);
    if (!h) return 0;
    PyObject *v = h == Py_None ? Py_NewRef(h) : PyObject_GetAttr(h, s_value);
    Py_DECREF(h);
    if (!v) return 0;
    *out = v == Py_None ? NULL : PyLong_AsVoidPtr(v);
    const int ok = v == Py_None || *out || !PyErr_Occurred();
    Py_DECREF(v);
    return ok;
}

/* The library may wait for the device (scratch that grows): other Python threads run meanwhile, as under ctypes. */
#define CALL(EXPR)                  \
    int status;                     \
    Py_BEGIN_ALLOW_THREADS          \
    status = (EXPR);                \
    Py_END_ALLOW_THREADS            \
    return finish(status)

static PyObject *gemv(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* out, matrix, v */
{
    size_t nv, no, ncols, nrows;
    void *m, *v, *out, *s;
    if (!expect(n, 3) || !numel(a[2], &nv) || !attr_size(a[1], s_ncols, &ncols)) return NULL;
    if (nv != ncols) return invalid("Gemv: dimension mismatch.");
    if (!numel(a[0], &no) || !attr_size(a[1], s_nrows, &nrows)) return NULL;
    if (no != nrows) return invalid("Gemv: dimension mismatch.");
    if (!handle(a[1], &m) || !f32(a[2], "v", &v) || !f32(a[0], "out", &out) || !current_stream(&s)) return NULL;
    CALL(((int (*)(void *, void *, void *, void *))fn[F_GEMV])(m, v, out, s));
}

static int two_dims(PyObject *t, size_t *d)   /* 0: error, 1: yes, 2: another number of dimensions */
{
    PyObject *s = PyObject_GetAttr(t, s_shape);
    if (!s) return 0;
    int r = 2;
    if (PyTuple_Check(s) && PyTuple_GET_SIZE(s) == 2) {
        d[0] = PyLong_AsSize_t(PyTuple_GET_ITEM(s, 0));
        d[1] = PyLong_AsSize_t(PyTuple_GET_ITEM(s, 1));
        r = PyErr_Occurred() ? 0 : 1;
    }
    Py_DECREF(s);
    return r;
}

static PyObject *gemm(PyObject *const *a, Py_ssize_t n, int which)   /* out, tiles, v */
{
    size_t dv[2], dout[2], ncols, nrows;
    void *m, *v, *out, *s;
    if (!expect(n, 3)) return NULL;
    const int tv = two_dims(a[2], dv), to = tv ? two_dims(a[0], dout) : 0;
    if (!tv || !to || !attr_size(a[1], s_ncols, &ncols) || !attr_size(a[1], s_nrows, &nrows)) return NULL;
    if (tv == 2 || to == 2 || dv[1] != ncols || dout[1] != nrows || dv[0] != dout[0]) return invalid("Gemm: dimension mismatch.");
    if (!handle(a[1], &m) || !f32(a[2], "v", &v) || !f32(a[0], "out", &out) || !current_stream(&s)) return NULL;
    CALL(((int (*)(void *, void *, size_t, void *, void *))fn[which])(m, v, dv[0], out, s));
}
static PyObject *gemm_q4k(PyObject *self, PyObject *const *a, Py_ssize_t n) { return gemm(a, n, F_GEMM_Q4K); }
static PyObject *gemm_q6k(PyObject *self, PyObject *const *a, Py_ssize_t n) { return gemm(a, n, F_GEMM_Q6K); }
static PyObject *gemm_q80(PyObject *self, PyObject *const *a, Py_ssize_t n) { return gemm(a, n, F_GEMM_Q80); }

static PyObject *rms_norm(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* result, value, weight, eps */
{
    size_t nv, nw, nr;
    void *r, *v, *w, *s;
    if (!expect(n, 4) || !numel(a[1], &nv) || !numel(a[2], &nw)) return NULL;
    if (nw != nv) return invalid("RmsNorm: dimension mismatch.");
    if (!numel(a[0], &nr)) return NULL;
    if (nr != nv) return invalid("RmsNorm: dimension mismatch.");
    const double eps = PyFloat_AsDouble(a[3]);
    if (eps == -1.0 && PyErr_Occurred()) return NULL;
    if (!f32(a[0], "result", &r) || !f32(a[1], "value", &v) || !f32(a[2], "weight", &w) || !current_stream(&s)) return NULL;
    CALL(((int (*)(void *, void *, void *, size_t, float, void *))fn[F_RMS_NORM])(r, v, w, nv, (float)eps, s));
}

/* Copies a parameter structure: of its own ctypes class or a derived one, whose first fields are the same. */
static int structure(PyObject *o, PyObject *type, const char *what, void *to, Py_ssize_t size)
{
    const int is = PyObject_IsInstance(o, type);
    if (is < 0) return 0;
    if (!is) {
        PyErr_SetString(PyExc_TypeError, what);
        return 0;
    }
    Py_buffer b;
    if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE)) return 0;
    const int fits = b.len >= size;
    if (fits) memcpy(to, b.buf, (size_t)size);
    PyBuffer_Release(&b);
    if (!fits) PyErr_SetString(PyExc_TypeError, what);
    return fits;
}

static PyObject *rope(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* variant, config structure, q, k */
{
    size_t nq, nk;
    void *q, *k, *s;
    if (!expect(n, 4)) return NULL;
    const long variant = PyLong_AsLong(a[0]);
    if (variant == -1 && PyErr_Occurred()) return NULL;
    struct { uint32_t head_size, kv_dim, pos; float base; } cfg;
    if (!structure(a[1], rope_config, "shape: expected a RoPEConfig", &cfg, sizeof(cfg))) return NULL;
    if (!f32(a[2], "in_out_q", &q) || !numel(a[2], &nq) || !f32(a[3], "in_out_k", &k) || !numel(a[3], &nk) || !current_stream(&s)) return NULL;
    CALL(((int (*)(int, const void *, void *, size_t, void *, size_t, void *))fn[F_ROPE])((int)variant, &cfg, q, nq, k, nk, s));
}

static PyObject *attention(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* params structure, q, keys, values, weights or None, xb */
{
    if (!expect(n, 6)) return NULL;
    struct { uint32_t seq_len, kv_dim, kv_mul, n_heads, head_size, pos; } p;
    if (!structure(a[0], attn_params, "params: expected BatchedMultiqueryAttentionParams", &p, sizeof(p))) return NULL;
    const size_t need = (size_t)p.seq_len * p.kv_dim;
    size_t nk, nv, nq, nx, na = 0;
    if (!numel(a[2], &nk) || !numel(a[3], &nv) || !numel(a[1], &nq) || !numel(a[5], &nx) || (a[4] != Py_None && !numel(a[4], &na))) return NULL;
    if (nk < need || nv < need || nq != (size_t)p.n_heads * p.head_size || nx != nq || (a[4] != Py_None && na < (size_t)p.n_heads * p.seq_len))
        return invalid("attention: dimension mismatch.");
    void *q, *k, *v, *w = NULL, *x, *s;
    if (!f32(a[1], "q", &q) || !f32(a[2], "key_cache", &k) || !f32(a[3], "value_cache", &v) || (a[4] != Py_None && !f32(a[4], "attn", &w)) ||
        !f32(a[5], "xb", &x) || !current_stream(&s))
        return NULL;
    CALL(((int (*)(const void *, void *, void *, void *, void *, void *, void *))fn[F_ATTENTION])(&p, q, k, v, w, x, s));
}

static PyObject *silu(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* h1, h2 */
{
    size_t n1, n2;
    void *x, *y, *s;
    if (!expect(n, 2) || !numel(a[0], &n1) || !numel(a[1], &n2)) return NULL;
    if (n1 != n2) return invalid("Silu: dimension mismatch.");
    if (!f32(a[0], "in_out_h1", &x) || !f32(a[1], "in_h2", &y) || !current_stream(&s)) return NULL;
    CALL(((int (*)(void *, void *, size_t, void *))fn[F_SILU])(x, y, n1, s));
}

static PyObject *op_assign(PyObject *self, PyObject *const *a, Py_ssize_t n)   /* variant, lhs, rhs */
{
    size_t n1, n2;
    void *x, *y, *s;
    if (!expect(n, 3) || !numel(a[1], &n1) || !numel(a[2], &n2)) return NULL;
    if (n1 != n2) return invalid("OpAssign: dimension mismatch.");
    const long variant = PyLong_AsLong(a[0]);
    if (variant == -1 && PyErr_Occurred()) return NULL;
    if (!f32(a[1], "lhs", &x) || !f32(a[2], "rhs", &y) || !current_stream(&s)) return NULL;
    CALL(((int (*)(int, void *, void *, size_t, void *))fn[F_OP_ASSIGN])((int)variant, x, y, n1, s));
}

#define FAST(NAME) { #NAME, (PyCFunction)(void (*)(void))NAME, METH_FASTCALL, NULL }
static PyMethodDef methods[] = {
    { "setup", setup, METH_VARARGS, NULL },
    FAST(gemv), FAST(gemm_q4k), FAST(gemm_q6k), FAST(gemm_q80), FAST(rms_norm), FAST(rope), FAST(attention), FAST(silu), FAST(op_assign),
    { NULL, NULL, 0, NULL },
};
static struct PyModuleDef module = { PyModuleDef_HEAD_INIT, "_dispatch", NULL, -1, methods, NULL, NULL, NULL, NULL };

PyMODINIT_FUNC PyInit__dispatch(void)
{
    struct { PyObject **at; const char *text; } names[] = {
        { &s_is_cuda, "is_cuda" }, { &s_dtype, "dtype" }, { &s_is_contiguous, "is_contiguous" }, { &s_data_ptr, "data_ptr" }, { &s_numel, "numel" },
        { &s_shape, "shape" }, { &s_h, "_h" }, { &s_value, "value" }, { &s_nrows, "nrows" }, { &s_ncols, "ncols" },
    };
    for (size_t i = 0; i < sizeof(names) / sizeof(names[0]); i++)
        if (!(*names[i].at = PyUnicode_InternFromString(names[i].text))) return NULL;
    PyObject *m = PyModule_Create(&module), *list = m ? PyTuple_New(F_COUNT) : NULL;
    for (Py_ssize_t i = 0; list && i < F_COUNT; i++) {
        PyObject *text = PyUnicode_FromString(entry[i]);
        if (!text) Py_CLEAR(list);
        else PyTuple_SET_ITEM(list, i, text);
    }
    if (!list || PyModule_AddObjectRef(m, "ENTRY_POINTS", list)) Py_CLEAR(m);
    Py_XDECREF(list);
    return m;
}
