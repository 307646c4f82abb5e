// The calls a decode step makes most often, as a CPython extension module over the C ABI (include/qk_moe.h).
//
// A call through ctypes converts eight arguments and looks three pointers up in Python: 2.4 us, as long as the host part of a
// kernel launch.  Here it is 0.4 us.  Arguments are what the ctypes signatures take; a pointer is None, an int, an object with
// data_ptr() (a torch tensor) or one with ptr (DevBuf).  Every function returns the C ABI's return code and runs without the GIL.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "../../include/qk_moe.h"

namespace {

PyObject *s_data_ptr, *s_ptr;   // interned names

bool pointer(PyObject* o, void** out) {
    if (PyLong_CheckExact(o)) { *out = PyLong_AsVoidPtr(o); return !PyErr_Occurred(); }
    if (o == Py_None) { *out = nullptr; return true; }
    PyObject* r = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!r && PyErr_ExceptionMatches(PyExc_AttributeError)) {
        PyErr_Clear();
        r = PyObject_GetAttr(o, s_ptr);
        if (!r && PyErr_ExceptionMatches(PyExc_AttributeError)) { PyErr_Clear(); r = PyNumber_Long(o); }
    }
    if (!r) return false;
    if (r == Py_None) *out = nullptr;
    else *out = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    return !PyErr_Occurred();
}
bool u32(PyObject* o, uint32_t* out) {
    *out = (uint32_t)PyLong_AsUnsignedLongMask(o);
    return !PyErr_Occurred();
}
bool f32(PyObject* o, float* out) {
    *out = (float)PyFloat_AsDouble(o);
    return !PyErr_Occurred();
}
bool count(const char* name, Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return true;
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, n);
    return false;
}
template <typename F>
PyObject* run(F f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

// (ctx, type, W, x, y, M, K, n)
PyObject* gemv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *c, *w, *x, *y;
    uint32_t type, M, K, rows;
    if (!count("gemv", n, 8) || !pointer(a[0], &c) || !u32(a[1], &type) || !pointer(a[2], &w) || !pointer(a[3], &x) || !pointer(a[4], &y) ||
        !u32(a[5], &M) || !u32(a[6], &K) || !u32(a[7], &rows)) return nullptr;
    return run([&] { return qkm_gemv((qkm_ctx*)c, type, w, (const float*)x, (float*)y, M, K, rows); });
}
// (ctx, index, x, n, y)
template <int (*F)(qkm_ctx*, uint32_t, const float*, uint32_t, float*)>
PyObject* rows_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *c, *x, *y;
    uint32_t index, rows;
    if (!count("call", n, 5) || !pointer(a[0], &c) || !u32(a[1], &index) || !pointer(a[2], &x) || !u32(a[3], &rows) || !pointer(a[4], &y)) return nullptr;
    return run([&] { return F((qkm_ctx*)c, index, (const float*)x, rows, (float*)y); });
}
// (ctx, first, count, x, n, y)
template <int (*F)(qkm_ctx*, uint32_t, uint32_t, const float*, uint32_t, float*)>
PyObject* stack_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *c, *x, *y;
    uint32_t first, layers, rows;
    if (!count("call", n, 6) || !pointer(a[0], &c) || !u32(a[1], &first) || !u32(a[2], &layers) || !pointer(a[3], &x) || !u32(a[4], &rows) ||
        !pointer(a[5], &y)) return nullptr;
    return run([&] { return F((qkm_ctx*)c, first, layers, (const float*)x, rows, (float*)y); });
}
// (ctx, logits, n_rows, n, tok)
PyObject* argmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *c, *l, *t;
    uint32_t rows, len;
    if (!count("argmax", n, 5) || !pointer(a[0], &c) || !pointer(a[1], &l) || !u32(a[2], &rows) || !u32(a[3], &len) || !pointer(a[4], &t)) return nullptr;
    return run([&] { return qkm_argmax((qkm_ctx*)c, (const float*)l, rows, len, (uint32_t*)t); });
}
// (ctx, layer, resid, attn_out, w_post, w_next, n, eps, resid_out, xn_next)
PyObject* layer_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *c, *p[6];
    uint32_t layer, rows;
    float eps;
    if (!count("layer_step", n, 10) || !pointer(a[0], &c) || !u32(a[1], &layer) || !pointer(a[2], &p[0]) || !pointer(a[3], &p[1]) || !pointer(a[4], &p[2]) ||
        !pointer(a[5], &p[3]) || !u32(a[6], &rows) || !f32(a[7], &eps) || !pointer(a[8], &p[4]) || !pointer(a[9], &p[5])) return nullptr;
    return run([&] {
        return qkm_moe_layer_step((qkm_ctx*)c, layer, (const float*)p[0], (const float*)p[1], (const float*)p[2], (const float*)p[3], rows, eps,
                                  (float*)p[4], (float*)p[5]);
    });
}

#define FAST(f) ((PyCFunction)(void (*)(void))(f))
PyMethodDef methods[] = {
    {"gemv", FAST(gemv), METH_FASTCALL, nullptr},
    {"moe_decode", FAST(rows_call<qkm_moe_decode>), METH_FASTCALL, nullptr},
    {"moe_prefill", FAST(rows_call<qkm_moe_prefill>), METH_FASTCALL, nullptr},
    {"dense_gemm", FAST(rows_call<qkm_dense_gemm>), METH_FASTCALL, nullptr},
    {"moe_decode_stack", FAST(stack_call<qkm_moe_decode_stack>), METH_FASTCALL, nullptr},
    {"moe_decode_stack_host", FAST(stack_call<qkm_moe_decode_stack_host>), METH_FASTCALL, nullptr},
    {"argmax", FAST(argmax), METH_FASTCALL, nullptr},
    {"moe_layer_step", FAST(layer_step), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "qkm_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_qkm_calls(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_ptr = PyUnicode_InternFromString("ptr");
    return s_data_ptr && s_ptr ? PyModule_Create(&module) : nullptr;
}
