/* Python binding of the entry points that a decode or draft step calls many times: vector-call functions
 * over plain integers (addresses, sizes, flags; None is a null pointer), one per C entry point, returning
 * its status. A ctypes call with seventeen converted arguments takes longer than the launches it makes
 * (about 9 us against 2). Everything else is bound through ctypes (lib.py). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "frx.h"

#define MAX_ARGS 24
typedef long long i64;

static int ints(PyObject* const* a, Py_ssize_t n, Py_ssize_t want, i64* v) {
    if (n != want) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
        return -1;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
        if (a[i] == Py_None) {
            v[i] = 0;
            continue;
        }
        v[i] = PyLong_AsLongLong(a[i]);
        if (v[i] == -1 && PyErr_Occurred()) return -1;
    }
    return 0;
}

#define P(i) ((void*)(intptr_t)v[i])
#define S(i) ((frx_stream_t)(intptr_t)v[i])
#define I(i) ((int)v[i])
#define Z(i) ((size_t)v[i])
#define BIND(name, nargs, call)                                                    \
    static PyObject* py_##name(PyObject* self, PyObject* const* a, Py_ssize_t n) { \
        i64 v[MAX_ARGS];                                                           \
        (void)self;                                                                \
        if (ints(a, n, nargs, v)) return NULL;                                     \
        int rc;                                                                    \
        Py_BEGIN_ALLOW_THREADS                                                     \
        rc = call;                                                                 \
        Py_END_ALLOW_THREADS                                                       \
        return PyLong_FromLong(rc);                                                \
    }

BIND(route_topk, 10, frx_route_topk(S(0), P(1), I(2), I(3), I(4), P(5), P(6), P(7), P(8), I(9)))
BIND(router_logits, 9, frx_router_logits(S(0), P(1), P(2), P(3), I(4), I(5), I(6), P(7), P(8)))
BIND(quantize_q8, 6, frx_quantize_q8(S(0), P(1), I(2), I(3), P(4), P(5)))
BIND(moe_decode, 17, frx_moe_decode(P(0), Z(1), I(2), P(3), I(4), I(5), P(6), P(7), P(8), P(9), I(10), I(11), P(12), P(13), P(14), Z(15), S(16)))
BIND(moe_decode_static, 14, frx_moe_decode_static(P(0), Z(1), I(2), P(3), I(4), I(5), P(6), P(7), P(8), P(9), I(10), I(11), P(12), S(13)))
BIND(moe_layer, 17, frx_moe_layer(P(0), Z(1), I(2), P(3), I(4), I(5), P(6), P(7), P(8), I(9), I(10), P(11), P(12), P(13), P(14), Z(15), S(16)))
BIND(moe_hits, 11, frx_moe_hits(P(0), P(1), I(2), P(3), I(4), I(5), P(6), Z(7), P(8), S(9), I(10)))
BIND(moe_combine, 10, frx_moe_combine(P(0), P(1), P(2), P(3), P(4), P(5), I(6), I(7), I(8), S(9)))
BIND(chain_rmsnorm_unit, 6, frx_chain_rmsnorm_unit(P(0), P(1), P(2), I(3), I(4), S(5)))
BIND(gemv_quantize_q8_1, 5, frx_gemv_quantize_q8_1(P(0), v[1], I(2), P(3), S(4)))
BIND(gemv_swiglu_q8_1, 6, frx_gemv_swiglu_q8_1(P(0), P(1), v[2], I(3), P(4), S(5)))
BIND(gemv_moe_q, 13, frx_gemv_moe_q((uint32_t)v[0], P(1), P(2), P(3), P(4), P(5), I(6), I(7), v[8], v[9], v[10], I(11), S(12)))
BIND(gemv_moe_q2_0, 11, frx_gemv_moe_q2_0(P(0), P(1), P(2), P(3), P(4), I(5), v[6], v[7], v[8], I(9), S(10)))
BIND(gemv_matvec, 9, frx_gemv_matvec((uint32_t)v[0], P(1), P(2), P(3), v[4], v[5], I(6), P(7), S(8)))
BIND(gemm_moe_prepare, 12, frx_gemm_moe_prepare(P(0), (uint32_t)v[1], I(2), P(3), I(4), P(5), v[6], I(7), v[8], P(9), Z(10), S(11)))
BIND(gemm_moe_run, 6, frx_gemm_moe_run(P(0), P(1), v[2], P(3), v[4], S(5)))

#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {ENTRY(route_topk),
                                ENTRY(router_logits),
                                ENTRY(quantize_q8),
                                ENTRY(moe_decode),
                                ENTRY(moe_decode_static),
                                ENTRY(moe_layer),
                                ENTRY(moe_hits),
                                ENTRY(moe_combine),
                                ENTRY(chain_rmsnorm_unit),
                                ENTRY(gemv_quantize_q8_1),
                                ENTRY(gemv_swiglu_q8_1),
                                ENTRY(gemv_moe_q),
                                ENTRY(gemv_moe_q2_0),
                                ENTRY(gemv_matvec),
                                ENTRY(gemm_moe_prepare),
                                ENTRY(gemm_moe_run),
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_frxpy", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__frxpy(void) { return PyModule_Create(&module); }
