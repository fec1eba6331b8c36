// CPython side of the calls that programs make once per matrix: the Python binding's ctypes route spends about a microsecond per
// call on converting six arguments, as long as a small product takes on the GPU.  A tensor argument is anything with data_ptr()
// (torch), a .ctypes.data (numpy), an integer address or None.  Only argument passing lives here; status codes are
// returned as they are and turned into exceptions by the binding.
// Only the limited API of Python 3.10 is used, so one build serves every interpreter from there on; where it cannot be loaded, or was not built, the
// binding makes the same calls through ctypes.
#define PY_SSIZE_T_CLEAN
#define Py_LIMITED_API 0x030A0000
#include <Python.h>

#include "minfer_b200.h"

namespace {

PyObject *s_data_ptr, *s_ctypes, *s_data, *s_shape;

// address of a tensor-like argument; false with a Python error set
bool address(PyObject* o, void** out) {
    if (o == Py_None) { *out = nullptr; return true; }
    if (PyLong_Check(o)) { *out = PyLong_AsVoidPtr(o); return !PyErr_Occurred(); }
    PyObject* v = PyObject_CallMethodObjArgs(o, s_data_ptr, static_cast<PyObject*>(nullptr));
    if (!v && PyErr_ExceptionMatches(PyExc_AttributeError)) {
        PyErr_Clear();
        PyObject* c = PyObject_GetAttr(o, s_ctypes);
        if (c) { v = PyObject_GetAttr(c, s_data); Py_DECREF(c); }
    }
    if (!v) return false;
    *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    return !PyErr_Occurred();
}
bool integer(PyObject* o, long long* out) { *out = PyLong_AsLongLong(o); return !(*out == -1 && PyErr_Occurred()); }
bool count(Py_ssize_t got, Py_ssize_t want, const char* name) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
    return false;
}

// quant_q8(ctx, x, xq, xd, n or None: the last dimension of x, M)
PyObject* quant_q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *ctx, *x, *xq, *xd; long long len, M;
    if (!count(n, 6, "quant_q8") || !address(a[0], &ctx) || !address(a[1], &x) || !address(a[2], &xq) || !address(a[3], &xd) || !integer(a[5], &M)) return nullptr;
    if (a[4] == Py_None) {
        PyObject* shape = PyObject_GetAttr(a[1], s_shape);
        if (!shape) return nullptr;
        PyObject* last = PySequence_GetItem(shape, -1);
        Py_DECREF(shape);
        if (!last) return nullptr;
        const bool ok = integer(last, &len);
        Py_DECREF(last);
        if (!ok) return nullptr;
    } else if (!integer(a[4], &len)) return nullptr;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = mi_quant_q8(static_cast<mi_ctx*>(ctx), static_cast<const float*>(x), len, (int)M, static_cast<int8_t*>(xq), static_cast<uint16_t*>(xd));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(st);
}

// gemv_q4_q8(ctx, w, xq, xd, bias, y, ksplit, variant)
PyObject* gemv_q4_q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *ctx, *w, *xq, *xd, *bias, *y; long long ks, v;
    if (!count(n, 8, "gemv_q4_q8") || !address(a[0], &ctx) || !address(a[1], &w) || !address(a[2], &xq) || !address(a[3], &xd) || !address(a[4], &bias) ||
        !address(a[5], &y) || !integer(a[6], &ks) || !integer(a[7], &v)) return nullptr;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = mi_gemv_q4_q8_ex(static_cast<mi_ctx*>(ctx), static_cast<const mi_weight*>(w), static_cast<const int8_t*>(xq), static_cast<const uint16_t*>(xd),
                          static_cast<const float*>(bias), static_cast<float*>(y), (int)ks, (int)v);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(st);
}

// gemm_q4_q8(ctx, w, xq, xd, M, bias, y)
PyObject* gemm_q4_q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *ctx, *w, *xq, *xd, *bias, *y; long long M;
    if (!count(n, 7, "gemm_q4_q8") || !address(a[0], &ctx) || !address(a[1], &w) || !address(a[2], &xq) || !address(a[3], &xd) || !integer(a[4], &M) ||
        !address(a[5], &bias) || !address(a[6], &y)) return nullptr;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = mi_gemm_q4_q8(static_cast<mi_ctx*>(ctx), static_cast<const mi_weight*>(w), static_cast<const int8_t*>(xq), static_cast<const uint16_t*>(xd), (int)M,
                       static_cast<const float*>(bias), static_cast<float*>(y));
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(st);
}

PyMethodDef methods[] = {
    {"quant_q8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(quant_q8)), METH_FASTCALL, nullptr},
    {"gemv_q4_q8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemv_q4_q8)), METH_FASTCALL, nullptr},
    {"gemm_q4_q8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm_q4_q8)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "minfer_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_minfer_fastcall(void) {
    s_data_ptr = PyUnicode_InternFromString("data_ptr"); s_ctypes = PyUnicode_InternFromString("ctypes");
    s_data = PyUnicode_InternFromString("data"); s_shape = PyUnicode_InternFromString("shape");
    return s_data_ptr && s_ctypes && s_data && s_shape ? PyModule_Create(&module) : nullptr;
}
