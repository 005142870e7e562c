/* Node: the part of `Tensor` that records a graph, as a CPython type over the rcu_lazy_* entry points.
 *
 * A model's schedule() is a few hundred builder calls and the device idles until it is through.  Through ctypes a call costs about
 * 2.6 us (argument conversion, a c_void_p and a reference to it, the status check, a Python object and its __del__); here it costs
 * 0.2.  Measured on a B200's host (us before the resolve): eight Phi-3 layers over 1000 tokens (461 nodes) 923 -> 115, Whisper's
 * encoder (230 nodes) 350 -> 58.
 *
 * The library is the one that ctypes has loaded (bind(path)): the type holds function pointers, no state of its own.
 * Methods take their arguments by position or by name, as the Python methods that they stand in for. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <dlfcn.h>

#include "../../include/ratchet_cuda.h"

typedef struct {
    PyObject_HEAD
    PyObject* dev;
    rcu_lazy* h;
} Node;

static PyTypeObject NodeType;

#define FUNCTIONS(X)                                                                                                        \
    X(release) X(retain) X(info) X(strong_count) X(binary) X(unary) X(cast) X(norm) X(softmax) X(rope) X(matmul) X(conv1d)  \
    X(view) X(slice) X(permute) X(broadcast) X(index_select) X(cache) X(linear) X(norm_rows) X(stream_rows) X(post_norm)    \
    X(bitcast) X(rotary_angles) X(norm_rotary) X(kv_append) X(grouped_attention) X(glu) X(rotary) X(lightning)              \
    X(latent_append) X(window_attention)
#define X(name) static __typeof__(&rcu_lazy_##name) p_##name;
FUNCTIONS(X)
#undef X

static PyObject *s_handle, *s_check;
static int bound;

/* ------------------------------------------------------------------------------------------------ arguments */
static int as_node(PyObject* o, rcu_lazy** out) {          /* None: no tensor */
    if (o == NULL || o == Py_None) {
        *out = NULL;
        return 1;
    }
    if (!PyObject_TypeCheck(o, &NodeType)) {
        PyErr_Format(PyExc_TypeError, "a tensor is expected, not %.80s", Py_TYPE(o)->tp_name);
        return 0;
    }
    *out = ((Node*)o)->h;
    return 1;
}

static int as_word(PyObject* o, uint64_t* out) {           /* whole numbers wrap to the width of the C argument, as ctypes has it */
    if (PyLong_Check(o)) {
        *out = PyLong_AsUnsignedLongLongMask(o);
    } else {
        PyObject* i = PyNumber_Index(o);
        if (!i) return 0;
        *out = PyLong_AsUnsignedLongLongMask(i);
        Py_DECREF(i);
    }
    return !(*out == (uint64_t)-1 && PyErr_Occurred());
}

static int as_float(PyObject* o, float* out) {
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) return 0;
    *out = (float)d;
    return 1;
}

/* Whole numbers of a sequence (`convert`: int(entry) of any); entries beyond `cap` are counted, not stored (no rank is that large: the library
 * refuses).  A tuple of its own: converting an entry may run code that changes a list. */
static int as_words(PyObject* seq, int convert, uint64_t* out, Py_ssize_t cap, Py_ssize_t* n) {
    PyObject* f = PySequence_Tuple(seq);
    if (!f) return 0;
    *n = PyTuple_GET_SIZE(f);
    int ok = 1;
    for (Py_ssize_t i = 0; ok && i < *n && i < cap; ++i) {
        PyObject* o = PyTuple_GET_ITEM(f, i);
        if (PyLong_Check(o)) {
            out[i] = PyLong_AsUnsignedLongLongMask(o);
        } else {
            PyObject* w = convert ? PyNumber_Long(o) : PyNumber_Index(o);
            if (!w) { ok = 0; break; }
            out[i] = PyLong_AsUnsignedLongLongMask(w);
            Py_DECREF(w);
        }
        if (out[i] == (uint64_t)-1 && PyErr_Occurred()) ok = 0;
    }
    Py_DECREF(f);
    return ok;
}

/* positional and named arguments into out[count]; those not given stay NULL, the first `required` must be there */
static int gather(const char* fn, PyObject* const* a, Py_ssize_t n, PyObject* kw, const char* const* names, int count, int required, PyObject** out) {
    if (n > count) {
        PyErr_Format(PyExc_TypeError, "%s() takes at most %d arguments (%zd given)", fn, count, n);
        return 0;
    }
    for (int i = 0; i < count; ++i) out[i] = i < n ? a[i] : NULL;
    if (kw) {
        const Py_ssize_t m = PyTuple_GET_SIZE(kw);
        for (Py_ssize_t k = 0; k < m; ++k) {
            PyObject* name = PyTuple_GET_ITEM(kw, k);
            int i = 0;
            while (i < count && PyUnicode_CompareWithASCIIString(name, names[i]) != 0) ++i;
            if (i == count || out[i]) {
                PyErr_Format(PyExc_TypeError, i == count ? "%s() got an unexpected argument %R" : "%s() got multiple values for argument %R", fn, name);
                return 0;
            }
            out[i] = a[n + k];
        }
    }
    for (int i = 0; i < required; ++i)
        if (!out[i]) {
            PyErr_Format(PyExc_TypeError, "%s() missing argument '%s'", fn, names[i]);
            return 0;
        }
    return 1;
}

/* a tensor of self's class and device over `h`, or the device's error for `st` */
static PyObject* finish(Node* self, rcu_status st, rcu_lazy* h) {
    if (st != RCU_OK) {
        PyObject* code = PyLong_FromLong((long)st);
        if (!code) return NULL;
        PyObject* r = PyObject_CallMethodOneArg(self->dev, s_check, code);
        Py_DECREF(code);
        if (r) {
            Py_DECREF(r);
            PyErr_Format(PyExc_RuntimeError, "status %d", (int)st);
        }
        return NULL;
    }
    PyTypeObject* t = Py_TYPE(self);
    Node* o = (Node*)t->tp_alloc(t, 0);
    if (!o) {
        p_release(h);
        return NULL;
    }
    o->dev = Py_NewRef(self->dev);
    o->h = h;
    return (PyObject*)o;
}

/* ------------------------------------------------------------------------------------------------ lifetime */
static int open_handle(Node* self) {                       /* a closed device has already dropped everything */
    PyObject* d = PyObject_GetAttr(self->dev, s_handle);
    const int open = d ? PyObject_IsTrue(d) : -1;
    Py_XDECREF(d);
    return open;
}

static int drop(Node* self) {
    rcu_lazy* h = self->h;
    if (!h) return 0;
    const int open = open_handle(self);
    self->h = NULL;
    if (open > 0) p_release(h);
    return open < 0 ? -1 : 0;
}

static void node_dealloc(Node* self) {
    if (self->h) {
        PyObject *type, *value, *trace;
        PyErr_Fetch(&type, &value, &trace);
        if (drop(self) < 0) PyErr_Clear();
        PyErr_Restore(type, value, trace);
    }
    Py_CLEAR(self->dev);
    Py_TYPE(self)->tp_free((PyObject*)self);
}

static PyObject* node_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
    static char* names[] = {"dev", "handle", NULL};
    PyObject *dev, *handle;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "OO", names, &dev, &handle)) return NULL;
    if (!bound) {                                          /* no handle can come from anywhere else, and no method could run */
        PyErr_SetString(PyExc_RuntimeError, "the runtime library has not been loaded (capi.lib())");
        return NULL;
    }
    PyObject* value = PyLong_Check(handle) || handle == Py_None ? Py_NewRef(handle) : PyObject_GetAttrString(handle, "value");     /* a c_void_p */
    if (!value) return NULL;
    void* h = value == Py_None ? NULL : PyLong_AsVoidPtr(value);
    Py_DECREF(value);
    if (!h && PyErr_Occurred()) return NULL;
    Node* o = (Node*)type->tp_alloc(type, 0);
    if (!o) return NULL;
    o->dev = Py_NewRef(dev);
    o->h = (rcu_lazy*)h;
    return (PyObject*)o;
}

static int node_init(PyObject* self, PyObject* args, PyObject* kw) { (void)self; (void)args; (void)kw; return 0; }

static PyObject* node_consume(Node* self, PyObject* unused) {
    (void)unused;
    if (drop(self) < 0) return NULL;
    Py_RETURN_NONE;
}

static PyObject* node_clone(Node* self, PyObject* unused) {
    (void)unused;
    p_retain(self->h);
    return finish(self, RCU_OK, self->h);
}

static PyObject* node_handle(Node* self, void* unused) {
    (void)unused;
    if (!self->h) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(self->h);
}

static PyObject* node_strong_count(Node* self, PyObject* u) { (void)u; return PyLong_FromUnsignedLong(p_strong_count(self->h)); }

/* ------------------------------------------------------------------------------------------------ introspection */
static int info(Node* self, rcu_tensor* t) {
    memset(t, 0, sizeof *t);
    return p_info(self->h, t);
}

static PyObject* node_shape(Node* self, PyObject* u) {
    (void)u;
    rcu_tensor t;
    info(self, &t);
    PyObject* out = PyTuple_New(t.rank);
    for (uint32_t i = 0; out && i < t.rank; ++i) {
        PyObject* v = PyLong_FromUnsignedLongLong(t.shape[i]);
        if (!v) { Py_DECREF(out); return NULL; }
        PyTuple_SET_ITEM(out, i, v);
    }
    return out;
}
static PyObject* node_rank(Node* self, PyObject* u) { (void)u; rcu_tensor t; info(self, &t); return PyLong_FromUnsignedLong(t.rank); }
static PyObject* node_dt(Node* self, PyObject* u) { (void)u; rcu_tensor t; info(self, &t); return PyLong_FromLong(t.dt); }
static PyObject* node_resolved(Node* self, PyObject* u) { (void)u; rcu_tensor t; return PyBool_FromLong(info(self, &t)); }
static PyObject* node_data_ptr(Node* self, PyObject* u) { (void)u; rcu_tensor t; info(self, &t); return PyLong_FromVoidPtr(t.data); }

/* ------------------------------------------------------------------------------------------------ builders */
#define METHOD(fn) static PyObject* node_##fn(Node* self, PyObject* const* a, Py_ssize_t n, PyObject* kw)
#define ARGS(fn, count, required, ...)                                       \
    static const char* const names[] = {__VA_ARGS__};                        \
    PyObject* v[count];                                                      \
    if (!gather(fn, a, n, kw, names, count, required, v)) return NULL;       \
    rcu_lazy* out = NULL
#define NODE(i) rcu_lazy* x##i; if (!as_node(v[i], &x##i)) return NULL
#define WORD(i) uint64_t w##i; if (!as_word(v[i], &w##i)) return NULL
#define REAL(i) float f##i; if (!as_float(v[i], &f##i)) return NULL
#define DONE(call)                 \
    do {                           \
        const rcu_status st = (call); \
        return finish(self, st, out); \
    } while (0)

#define BINARY(fn, op)                                                        \
    METHOD(fn) { ARGS(#fn, 1, 1, "other"); NODE(0); DONE(p_binary(op, self->h, x0, &out)); }
BINARY(add, RCU_ADD) BINARY(sub, RCU_SUB) BINARY(mul, RCU_MUL) BINARY(div, RCU_DIV)

#define UNARY(fn, op)                                                         \
    static PyObject* node_##fn(Node* self, PyObject* u) { (void)u; rcu_lazy* out = NULL; DONE(p_unary(op, self->h, &out)); }
UNARY(gelu, RCU_GELU) UNARY(tanh, RCU_TANH) UNARY(exp, RCU_EXP) UNARY(log, RCU_LOG) UNARY(sin, RCU_SIN) UNARY(cos, RCU_COS) UNARY(abs, RCU_ABS)
UNARY(sqrt, RCU_SQRT) UNARY(relu, RCU_RELU) UNARY(floor, RCU_FLOOR) UNARY(ceil, RCU_CEIL) UNARY(neg, RCU_NEG) UNARY(sigmoid, RCU_SIGMOID)
UNARY(silu, RCU_SILU)

static PyObject* node_full(Node* self, PyObject* u) { (void)u; rcu_lazy* out = NULL; DONE(p_cast(self->h, RCU_F32, &out)); }
static PyObject* node_half(Node* self, PyObject* u) { (void)u; rcu_lazy* out = NULL; DONE(p_cast(self->h, RCU_F16, &out)); }

METHOD(cast) { ARGS("cast", 1, 1, "dst_dt"); WORD(0); DONE(p_cast(self->h, (int32_t)w0, &out)); }
METHOD(layer_norm) {
    ARGS("layer_norm", 3, 3, "weight", "bias", "eps"); NODE(0); NODE(1); REAL(2);
    DONE(p_norm(RCU_LAYER_NORM, self->h, x0, x1, f2, 0, &out));
}
METHOD(rms_norm) { ARGS("rms_norm", 2, 2, "weight", "eps"); NODE(0); REAL(1); DONE(p_norm(RCU_RMS_NORM, self->h, x0, NULL, f1, 0, &out)); }
METHOD(group_norm) {
    ARGS("group_norm", 4, 4, "num_groups", "weight", "bias", "eps"); WORD(0); NODE(1); NODE(2); REAL(3);
    DONE(p_norm(RCU_GROUP_NORM, self->h, x1, x2, f3, (uint32_t)w0, &out));
}
METHOD(conv1d) {
    ARGS("conv1d", 4, 4, "weight", "bias", "stride", "padding"); NODE(0); NODE(1); WORD(2); WORD(3);
    DONE(p_conv1d(self->h, x0, x1, (uint32_t)w2, (uint32_t)w3, &out));
}
METHOD(softmax) { ARGS("softmax", 1, 1, "dim"); WORD(0); DONE(p_softmax(self->h, (uint32_t)w0, &out)); }
METHOD(rope) { ARGS("rope", 3, 3, "dim", "base", "offset"); WORD(0); REAL(1); WORD(2); DONE(p_rope(self->h, (uint32_t)w0, f1, (uint32_t)w2, &out)); }

static int as_flag(PyObject* o, int* out) {               /* int(o); not given: 0 */
    *out = 0;
    if (!o || o == Py_False) return 1;
    if (o == Py_True) { *out = 1; return 1; }
    PyObject* i = PyNumber_Long(o);
    if (!i) return 0;
    *out = (int)PyLong_AsUnsignedLongMask(i);
    Py_DECREF(i);
    return !PyErr_Occurred();
}
METHOD(matmul) {
    ARGS("matmul", 3, 1, "rhs", "trans_lhs", "trans_rhs"); NODE(0);
    int tl, tr;
    if (!as_flag(v[1], &tl) || !as_flag(v[2], &tr)) return NULL;
    DONE(p_matmul(self->h, x0, NULL, tl, tr, 0, &out));
}
METHOD(gemm) {
    ARGS("gemm", 5, 5, "rhs", "bias", "trans_lhs", "trans_rhs", "trans_out"); NODE(0); NODE(1);
    int tl, tr, to;
    if (!as_flag(v[2], &tl) || !as_flag(v[3], &tr) || !as_flag(v[4], &to)) return NULL;
    DONE(p_matmul(self->h, x0, x1, tl, tr, to, &out));
}
METHOD(slice) {
    /* a list of (start, stop) pairs, one per dimension; other forms go through the general method */
    ARGS("slice", 1, 1, "ranges");
    uint64_t start[RCU_MAX_RANK], stop[RCU_MAX_RANK];
    rcu_tensor t;
    info(self, &t);
    int plain = PyList_CheckExact(v[0]) && PyList_GET_SIZE(v[0]) == (Py_ssize_t)t.rank;
    for (uint32_t i = 0; plain && i < t.rank; ++i) {
        PyObject* r = PyList_GET_ITEM(v[0], i);
        plain = PyTuple_CheckExact(r) && PyTuple_GET_SIZE(r) == 2 && PyLong_CheckExact(PyTuple_GET_ITEM(r, 0)) && PyLong_CheckExact(PyTuple_GET_ITEM(r, 1));
        if (!plain) break;
        start[i] = PyLong_AsUnsignedLongLongMask(PyTuple_GET_ITEM(r, 0));
        stop[i] = PyLong_AsUnsignedLongLongMask(PyTuple_GET_ITEM(r, 1));
    }
    if (!plain) return PyObject_CallMethod((PyObject*)self, "_slice", "(O)", v[0]);
    DONE(p_slice(self->h, start, stop, &out));
}
METHOD(view) {
    ARGS("view", 1, 1, "shape");
    uint64_t s[RCU_MAX_RANK];
    Py_ssize_t rank;
    if (!as_words(v[0], 1, s, RCU_MAX_RANK, &rank)) return NULL;
    DONE(p_view(self->h, (uint32_t)rank, s, &out));
}
METHOD(broadcast_to) {
    ARGS("broadcast_to", 1, 1, "shape");
    uint64_t s[RCU_MAX_RANK];
    Py_ssize_t rank;
    if (!as_words(v[0], 1, s, RCU_MAX_RANK, &rank)) return NULL;
    DONE(p_broadcast(self->h, (uint32_t)rank, s, &out));
}
METHOD(permute) {
    ARGS("permute", 1, 1, "dims");
    uint64_t s[RCU_MAX_RANK];
    uint32_t p[RCU_MAX_RANK];
    Py_ssize_t rank;
    rcu_tensor t;
    info(self, &t);
    if (!as_words(v[0], 0, s, RCU_MAX_RANK, &rank)) return NULL;
    if (rank != (Py_ssize_t)t.rank) return PyObject_CallMethod((PyObject*)self, "_permute_rank", NULL);
    for (Py_ssize_t i = 0; i < rank; ++i) p[i] = (uint32_t)s[i];
    DONE(p_permute(self->h, p, &out));
}
METHOD(cache) {
    ARGS("cache", 3, 3, "source", "dim", "offset"); NODE(0); WORD(1); WORD(2);
    DONE(p_cache(self->h, x0, (uint32_t)w1, (uint32_t)w2, &out));
}
METHOD(index_select) { ARGS("index_select", 2, 2, "indices", "dim"); NODE(0); WORD(1); DONE(p_index_select(self->h, x0, (uint32_t)w1, &out)); }

/* ops of models with a 32-bit residual stream: the _ forms take every argument, the Python methods fill in the defaults */
#define POSITIONAL(fn, count)                                                                              \
    PyObject* const* v = a;                                                                                \
    rcu_lazy* out = NULL;                                                                                  \
    if (n != (count) || kw) {                                                                              \
        PyErr_Format(PyExc_TypeError, "%s() takes %d positional arguments", fn, count);                    \
        return NULL;                                                                                       \
    }
METHOD(_linear) {       /* x, x_col, bias, act, act_cols, act_param, resid, alpha, dt */
    POSITIONAL("_linear", 9) NODE(0); WORD(1); NODE(2); WORD(3); WORD(4); REAL(5); NODE(6); REAL(7); WORD(8);
    DONE(p_linear(self->h, x0, (uint32_t)w1, x2, (int)w3, (uint32_t)w4, f5, x6, f7, (int32_t)w8, &out));
}
METHOD(_norm_rows) {    /* kind, col, scale, shift, gate, gate_col, eps, dt */
    POSITIONAL("_norm_rows", 8) WORD(0); WORD(1); NODE(2); NODE(3); NODE(4); WORD(5); REAL(6); WORD(7);
    DONE(p_norm_rows((int)w0, self->h, (uint32_t)w1, x2, x3, x4, (uint32_t)w5, f6, (int32_t)w7, &out));
}
METHOD(stream_rows) { ARGS("stream_rows", 1, 1, "copy_dt"); WORD(0); DONE(p_stream_rows(self->h, (int32_t)w0, &out)); }
METHOD(post_norm) {
    ARGS("post_norm", 4, 4, "y", "scale", "shift", "eps"); NODE(0); NODE(1); NODE(2); REAL(3);
    DONE(p_post_norm(self->h, x0, x1, x2, f3, &out));
}
METHOD(bitcast) { ARGS("bitcast", 1, 1, "dt"); WORD(0); DONE(p_bitcast(self->h, (int32_t)w0, &out)); }
METHOD(_glu) { POSITIONAL("_glu", 1) WORD(0); DONE(p_glu((int)w0, self->h, &out)); }
METHOD(_rotary) {       /* first, freqs, magnitude, position */
    POSITIONAL("_rotary", 4) WORD(0); NODE(1); REAL(2); WORD(3);
    DONE(p_rotary(self->h, (uint32_t)w0, x1, f2, (uint32_t)w3, &out));
}
METHOD(lightning) { ARGS("lightning", 2, 2, "decay_pow", "state"); NODE(0); NODE(1); DONE(p_lightning(self->h, x0, x1, &out)); }
METHOD(_latent_append) {        /* col, scale, eps, freqs, magnitude, position, ring, rows */
    POSITIONAL("_latent_append", 8) WORD(0); NODE(1); REAL(2); NODE(3); REAL(4); WORD(5); NODE(6); WORD(7);
    DONE(p_latent_append(self->h, (uint32_t)w0, x1, f2, x3, f4, (uint32_t)w5, x6, (uint32_t)w7, &out));
}
METHOD(window_attention) {
    ARGS("window_attention", 6, 6, "kv", "shared", "shared_col", "vdim", "window", "scale"); NODE(0); NODE(1); WORD(2); WORD(3); WORD(4); REAL(5);
    DONE(p_window_attention(self->h, x0, x1, (uint32_t)w2, (uint32_t)w3, (uint32_t)w4, f5, &out));
}
METHOD(rotary_angles) {
    ARGS("rotary_angles", 3, 3, "magnitude", "position", "tokens"); REAL(0); WORD(1); WORD(2);
    DONE(p_rotary_angles(self->h, f0, (uint32_t)w1, (uint32_t)w2, &out));
}
METHOD(_norm_rotary) {  /* col, heads, scale, eps, angles */
    POSITIONAL("_norm_rotary", 5) WORD(0); WORD(1); NODE(2); REAL(3); NODE(4);
    DONE(p_norm_rotary(self->h, (uint32_t)w0, (uint32_t)w1, x2, f3, x4, &out));
}
METHOD(_kv_append) {    /* col, kv_heads, scale, eps, angles, position, keep, ring, rows */
    POSITIONAL("_kv_append", 9) WORD(0); WORD(1); NODE(2); REAL(3); NODE(4); WORD(5); WORD(6); NODE(7); WORD(8);
    DONE(p_kv_append(self->h, (uint32_t)w0, (uint32_t)w1, x2, f3, x4, (uint32_t)w5, (uint32_t)w6, x7, (uint32_t)w8, &out));
}
METHOD(_grouped_attention) {    /* kv, sink, kv_heads, vdim, window, chunk, position, scale */
    POSITIONAL("_grouped_attention", 8) NODE(0); NODE(1); WORD(2); WORD(3); WORD(4); WORD(5); WORD(6); REAL(7);
    DONE(p_grouped_attention(self->h, x0, x1, (uint32_t)w2, (uint32_t)w3, (uint32_t)w4, (uint32_t)w5, (uint32_t)w6, f7, &out));
}

#define FAST(fn) {#fn, (PyCFunction)(void (*)(void))node_##fn, METH_FASTCALL | METH_KEYWORDS, NULL}
#define NOARGS(fn) {#fn, (PyCFunction)(void (*)(void))node_##fn, METH_NOARGS, NULL}
static PyMethodDef node_methods[] = {
    NOARGS(consume), NOARGS(clone), NOARGS(strong_count), NOARGS(shape), NOARGS(rank), NOARGS(dt), NOARGS(resolved), NOARGS(data_ptr),
    FAST(add), FAST(sub), FAST(mul), FAST(div),
    NOARGS(gelu), NOARGS(tanh), NOARGS(exp), NOARGS(log), NOARGS(sin), NOARGS(cos), NOARGS(abs), NOARGS(sqrt), NOARGS(relu), NOARGS(floor),
    NOARGS(ceil), NOARGS(neg), NOARGS(sigmoid), NOARGS(silu), NOARGS(full), NOARGS(half),
    FAST(cast), FAST(layer_norm), FAST(rms_norm), FAST(group_norm), FAST(conv1d), FAST(softmax), FAST(rope), FAST(matmul), FAST(gemm),
    FAST(slice), FAST(view), FAST(broadcast_to), FAST(permute), FAST(cache), FAST(index_select),
    FAST(_linear), FAST(_norm_rows), FAST(stream_rows), FAST(post_norm), FAST(bitcast), FAST(_glu), FAST(_rotary), FAST(lightning),
    FAST(_latent_append), FAST(window_attention), FAST(rotary_angles), FAST(_norm_rotary), FAST(_kv_append), FAST(_grouped_attention),
    {NULL, NULL, 0, NULL}};

static PyMemberDef node_members[] = {{"dev", T_OBJECT, offsetof(Node, dev), READONLY, NULL}, {NULL, 0, 0, 0, NULL}};
static PyGetSetDef node_getset[] = {{"_h", (getter)node_handle, NULL, "address of the lazy graph's node, None once consumed", NULL}, {NULL, NULL, NULL, NULL, NULL}};

static PyTypeObject NodeType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "ratchet_b200._graph.Node",
    .tp_basicsize = sizeof(Node),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE,
    .tp_dealloc = (destructor)node_dealloc,
    .tp_new = node_new,
    .tp_init = node_init,
    .tp_methods = node_methods,
    .tp_members = node_members,
    .tp_getset = node_getset,
};

/* bind(path): the entry points of the library that is loaded from `path` */
static PyObject* bind(PyObject* module, PyObject* path) {
    (void)module;
    const char* p = PyUnicode_AsUTF8(path);
    if (!p) return NULL;
    void* lib = dlopen(p, RTLD_NOW | RTLD_LOCAL);
    if (!lib) {
        PyErr_Format(PyExc_OSError, "%s", dlerror());
        return NULL;
    }
#define X(name)                                                               \
    if (!(p_##name = (__typeof__(p_##name))dlsym(lib, "rcu_lazy_" #name))) {   \
        PyErr_SetString(PyExc_AttributeError, "rcu_lazy_" #name);             \
        return NULL;                                                          \
    }
    FUNCTIONS(X)
#undef X
    bound = 1;
    Py_RETURN_NONE;
}

static PyMethodDef module_methods[] = {{"bind", bind, METH_O, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_graph", NULL, -1, module_methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__graph(void) {
    s_handle = PyUnicode_InternFromString("handle");
    s_check = PyUnicode_InternFromString("check");
    if (!s_handle || !s_check || PyType_Ready(&NodeType) < 0) return NULL;
    PyObject* m = PyModule_Create(&module_def);
    if (m && PyModule_AddObjectRef(m, "Node", (PyObject*)&NodeType) < 0) Py_CLEAR(m);
    return m;
}
