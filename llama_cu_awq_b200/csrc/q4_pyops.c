/* The op wrappers of llama_cu_awq_b200/ops.py as one C call each (module llama_cu_awq_b200._q4ops).
 *
 * Why: a token of a host program that calls the wrappers one by one is ~9 calls per layer. Through ctypes a call took 8 to 9 us
 * of Python time (argument boxing, the stream object, type conversions), more than most of the kernels it launches; here
 * it is one attribute-free argument walk plus the launch itself. The functions take the tensors' Python objects, ask
 * each for data_ptr(), and return the status code; ops.py turns a status that is not Q4_OK into the exception.
 * Only the CPython API and the C ABI of include/q4b200.h are used. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/q4b200.h"

static PyObject *s_data_ptr, *s_cuda_stream, *s_c;
static PyObject *f_raw_stream, *f_device; /* torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice */

/* An argument walk: every getter returns 0 / NULL and leaves a Python error set when the argument is not what it should be, and
 * does nothing at all behind an argument that failed (no Python code may run with an error set). */
static void* ptr_of(PyObject* o) { /* a tensor, or None */
    if (PyErr_Occurred() || o == Py_None) return NULL;
    PyObject* n = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!n) return NULL;
    void* p = PyLong_AsVoidPtr(n);
    Py_DECREF(n);
    return p;
}
static void* addr_of(PyObject* o) { /* an address (pinned host memory), or None */
    if (PyErr_Occurred() || o == Py_None) return NULL;
    if (!PyLong_Check(o)) {
        PyErr_Format(PyExc_TypeError, "an address is an int, not %.100s", Py_TYPE(o)->tp_name);
        return NULL;
    }
    return PyLong_AsVoidPtr(o);
}
static const q4_qweight* weight_of(PyObject* o) { /* QWeight.c, a ctypes q4_qweight; the QWeight keeps it */
    if (PyErr_Occurred()) return NULL;
    PyObject* c = PyObject_GetAttr(o, s_c);
    if (!c) return NULL;
    Py_buffer v;
    void* p = NULL;
    if (PyObject_GetBuffer(c, &v, PyBUF_SIMPLE) == 0) {
        if (v.len == (Py_ssize_t)sizeof(q4_qweight)) p = v.buf;
        else PyErr_SetString(PyExc_TypeError, "not a q4_qweight");
        PyBuffer_Release(&v);
    }
    Py_DECREF(c);
    return (const q4_qweight*)p;
}
static int int_of(PyObject* o) {
    if (PyErr_Occurred()) return 0;
    const long v = PyLong_AsLong(o);
    if (v > 2147483647L || v < -2147483647L - 1) {
        PyErr_SetString(PyExc_OverflowError, "size does not fit 32 bits");
        return 0;
    }
    return (int)v;
}
static int flag_of(PyObject* o) { return PyErr_Occurred() ? 0 : PyObject_IsTrue(o); }
static float float_of(PyObject* o) { return PyErr_Occurred() ? 0.f : (float)PyFloat_AsDouble(o); }
/* None: torch's current stream of the current device */
static void* stream_of(PyObject* o) {
    if (PyErr_Occurred()) return NULL;
    if (o != Py_None) {
        PyObject* n = PyObject_GetAttr(o, s_cuda_stream);
        if (!n) return NULL;
        void* p = PyLong_AsVoidPtr(n);
        Py_DECREF(n);
        return p;
    }
    PyObject* dev = PyObject_CallNoArgs(f_device);
    if (!dev) return NULL;
    PyObject* n = PyObject_CallOneArg(f_raw_stream, dev);
    Py_DECREF(dev);
    if (!n) return NULL;
    void* p = PyLong_AsVoidPtr(n);
    Py_DECREF(n);
    return p;
}

#define FN(name, count)                                                                   \
    static PyObject* py_##name(PyObject* self, PyObject* const* a, Py_ssize_t n) {        \
        (void)self;                                                                       \
        if (n != (count)) {                                                               \
            PyErr_Format(PyExc_TypeError, #name " takes %d arguments", (int)(count));     \
            return NULL;                                                                  \
        }
/* The call runs only when every argument converted, and without the interpreter lock: a launch blocks when the stream's
 * queue is full, and what the queue waits for may be another thread's launch (one thread per GPU, an all-reduce ahead). */
#define CALL(expr)                     \
    if (PyErr_Occurred()) return NULL; \
    int status;                        \
    Py_BEGIN_ALLOW_THREADS             \
    status = (expr);                   \
    Py_END_ALLOW_THREADS               \
    return PyLong_FromLong(status);    \
    }
#define P(i) ptr_of(a[i])
#define A(i) addr_of(a[i])
#define W(i) weight_of(a[i])
#define I(i) int_of(a[i])
#define F(i) float_of(a[i])
#define B(i) flag_of(a[i])
#define S(i) stream_of(a[i])

FN(rmsnorm, 5)
    void *s = S(0), *o = P(1), *x = P(2), *w = P(3);
    const int size = I(4);
    CALL(q4_rmsnorm(s, o, x, w, size))
FN(matmul_q4, 10)
    void *s = S(0), *o = P(1), *x = P(2);
    const q4_qweight* w = W(3);
    const int k = I(4), m = I(5), accum = B(6), g = I(7), loff = I(8);
    void* pos = P(9);
    CALL(q4_matmul_q4(s, o, x, w, k, m, accum, g, loff, pos))
FN(matmul_f16, 7)
    void *s = S(0), *o = P(1), *x = P(2), *w = P(3);
    const int k = I(4), m = I(5);
    const float alpha = F(6);
    CALL(q4_matmul_f16(s, o, x, w, k, m, alpha))
FN(qkv_matvec, 13)
    void *s = S(0), *q = P(1), *kc = P(2), *vc = P(3), *x = P(4);
    const q4_qweight *qw = W(5), *kw = W(6), *vw = W(7);
    const int k = I(8), m = I(9), kv = I(10), loff = I(11);
    void* pos = P(12);
    CALL(q4_qkv_matvec(s, q, kc, vc, x, qw, kw, vw, k, m, kv, loff, pos))
FN(ffn_matvec_silu, 7)
    void *s = S(0), *o = P(1), *x = P(2);
    const q4_qweight *gw = W(3), *uw = W(4);
    const int k = I(5), m = I(6);
    CALL(q4_ffn_matvec_silu(s, o, x, gw, uw, k, m))
FN(rope, 9)
    void *s = S(0), *q = P(1), *kc = P(2);
    const int nh = I(3), nkv = I(4), hs = I(5);
    void* pos = P(6);
    const int loff = I(7);
    const float theta = F(8);
    CALL(q4_rope(s, q, kc, nh, nkv, hs, pos, loff, theta))
FN(attention, 11)
    void *s = S(0), *o = P(1), *q = P(2), *kc = P(3), *vc = P(4), *scratch = P(5);
    const int nh = I(6), hs = I(7), mul = I(8), len = I(9);
    void* pos = P(10);
    CALL(q4_attention(s, o, q, kc, vc, scratch, nh, hs, mul, len, pos))
FN(embed, 6)
    void *s = S(0), *x = P(1), *table = P(2);
    const int dim = I(3);
    void *tok = A(4), *pos = P(5);
    CALL(q4_embed(s, x, table, dim, tok, pos))
FN(argmax, 7)
    void *s = S(0), *l = P(1);
    const int size = I(2);
    void *tok = A(3), *ppos = A(4), *dpos = P(5);
    const int write = B(6);
    CALL(q4_argmax(s, l, size, tok, ppos, dpos, write))
FN(sample_topp, 9)
    void *s = S(0), *l = P(1);
    const int size = I(2);
    const float t = F(3), topp = F(4), coin = F(5);
    void *tok = A(6), *ppos = A(7), *dpos = P(8);
    CALL(q4_sample_topp(s, l, size, t, topp, coin, tok, ppos, dpos))
FN(matmul_q4_batched, 10)
    void *s = S(0), *y = P(1), *x = P(2);
    const q4_qweight* w = W(3);
    void* wi = P(4);
    const int m = I(5), k = I(6), n2 = I(7);
    void* ws = P(8);
    const size_t bytes = PyErr_Occurred() ? 0 : PyLong_AsSize_t(a[9]);
    CALL(q4_matmul_q4_batched(s, y, x, w, wi, m, k, n2, ws, bytes))
FN(matmul_rows, 9)
    void *s = S(0), *y = P(1), *x = P(2);
    const q4_qweight* w = W(3);
    const int m = I(4), k = I(5), n2 = I(6);
    void* res = P(7);
    const float scale = F(8);
    CALL(q4_matmul_q4_rows(s, y, x, w, m, k, n2, res, scale))
FN(qkv_matmul_rows, 12)
    void *s = S(0), *q = P(1), *k = P(2), *v = P(3), *x = P(4);
    const q4_qweight *qw = W(5), *kw = W(6), *vw = W(7);
    const int m = I(8), in = I(9), out = I(10), kv = I(11);
    CALL(q4_qkv_matmul_rows(s, q, k, v, x, qw, kw, vw, m, in, out, kv))
FN(ffn_silu_rows, 8)
    void *s = S(0), *h = P(1), *x = P(2);
    const q4_qweight *gw = W(3), *uw = W(4);
    const int m = I(5), k = I(6), n2 = I(7);
    CALL(q4_ffn_silu_rows(s, h, x, gw, uw, m, k, n2))

#define M(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {M(rmsnorm), M(matmul_q4), M(matmul_f16), M(qkv_matvec), M(ffn_matvec_silu), M(rope), M(attention), M(embed), M(argmax),
                                M(sample_topp), M(matmul_q4_batched), M(matmul_rows), M(qkv_matmul_rows), M(ffn_silu_rows), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_q4ops", "The op wrappers of libq4b200.so, one C call each.", -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__q4ops(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    s_c = PyUnicode_InternFromString("c");
    PyObject* c = PyImport_ImportModule("torch._C");
    if (!c) return NULL;
    f_raw_stream = PyObject_GetAttrString(c, "_cuda_getCurrentRawStream");
    f_device = PyObject_GetAttrString(c, "_cuda_getDevice");
    Py_DECREF(c);
    if (!s_data_ptr || !s_cuda_stream || !s_c || !f_raw_stream || !f_device) return NULL;
    return PyModule_Create(&module);
}
