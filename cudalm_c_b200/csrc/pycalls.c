/* The entry points that a training step or a decode step calls many times, as plain C calls for Python: a ctypes call
 * converts each argument through its argtypes (about 2 us for ten), this takes them as they come.  A pointer argument is a
 * tensor (anything with data_ptr()), an address or None; a status other than 0 raises the exception class that
 * set_error_class() was given, with qlmb_last_error()'s text.  The remaining entry points are reached through ctypes. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include "../../include/qlm_b200.h"

static PyObject *error_class, *name_data_ptr;

/* The converters run in the order of the arguments.  After the first that failed the others do nothing: no Python code
 * may run with an exception set, and the caller is to see that one. */
static void *as_ptr(PyObject *o)
{
    if (o == Py_None || PyErr_Occurred()) return NULL;
    if (PyLong_CheckExact(o)) return PyLong_AsVoidPtr(o);
    PyObject *r = PyObject_CallMethodNoArgs(o, name_data_ptr);
    if (!r) return NULL;
    void *p = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    return p;
}
static int as_int(PyObject *o)
{
    if (PyErr_Occurred()) return 0;
    const long v = PyLong_AsLong(o);
    if (v == (int)v) return (int)v;
    PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int");
    return 0;
}
static float as_float(PyObject *o) { return PyErr_Occurred() ? 0.0f : (float)PyFloat_AsDouble(o); }
static unsigned long long as_u64(PyObject *o) { return PyErr_Occurred() ? 0 : PyLong_AsUnsignedLongLong(o); }

static PyObject *done(int rc)
{
    if (rc == 0) Py_RETURN_NONE;
    PyErr_Format(error_class ? error_class : PyExc_RuntimeError, "libqlm_b200 status %d: %s", rc, qlmb_last_error());
    return NULL;
}

/* N arguments: T converts them, the rest is the call */
#define CALL(NAME, N, T, ...)                                                                       \
    static PyObject *py_##NAME(PyObject *self, PyObject *const *a, Py_ssize_t n)                    \
    {                                                                                               \
        (void)self;                                                                                 \
        if (n != N) { PyErr_Format(PyExc_TypeError, #NAME " takes %d arguments, got %zd", N, n); return NULL; } \
        T;                                                                                          \
        if (PyErr_Occurred()) return NULL;                                                          \
        int rc;                                                                                     \
        Py_BEGIN_ALLOW_THREADS                                                                      \
        rc = qlmb_##NAME(__VA_ARGS__);                                                              \
        Py_END_ALLOW_THREADS                                                                        \
        return done(rc);                                                                            \
    }
#define ARG_P(k) void *const p##k = as_ptr(a[k])
#define ARG_I(k) const int i##k = as_int(a[k])
#define ARG_F(k) const float f##k = as_float(a[k])
#define ARG_U(k) const unsigned long long u##k = as_u64(a[k])

CALL(gemv_decode, 10, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_I(7); ARG_I(8); ARG_P(9),
     p0, p1, p2, p3, i4, i5, i6, i7, i8, p9)
CALL(linear_fwd, 11, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_I(7); ARG_P(8); ARG_I(9); ARG_P(10),
     p0, p1, p2, p3, i4, i5, i6, i7, p8, i9, p10)
CALL(linear_dgrad, 11, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_I(7); ARG_F(8); ARG_I(9); ARG_P(10),
     p0, p1, p2, p3, i4, i5, i6, i7, f8, i9, p10)
CALL(linear_wgrad, 10, ARG_P(0); ARG_P(1); ARG_P(2); ARG_I(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_F(7); ARG_I(8); ARG_P(9),
     p0, p1, p2, i3, i4, i5, i6, f7, i8, p9)
CALL(gemm_nt, 9, ARG_P(0); ARG_I(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_F(7); ARG_P(8),
     p0, i1, p2, p3, i4, i5, i6, f7, p8)
CALL(embed, 7, ARG_P(0); ARG_I(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_P(6), p0, i1, p2, p3, i4, i5, p6)
CALL(rmsnorm_fwd, 9, ARG_P(0); ARG_I(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_P(5); ARG_I(6); ARG_I(7); ARG_P(8),
     p0, i1, p2, p3, i4, p5, i6, i7, p8)
CALL(rmsnorm_bwd, 14, ARG_P(0); ARG_I(1); ARG_I(2); ARG_P(3); ARG_P(4); ARG_P(5); ARG_I(6); ARG_P(7); ARG_P(8); ARG_P(9); ARG_I(10);
     ARG_I(11); ARG_I(12); ARG_P(13), p0, i1, i2, p3, p4, p5, i6, p7, p8, p9, i10, i11, i12, p13)
CALL(rope, 10, ARG_P(0); ARG_I(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_I(6); ARG_I(7); ARG_I(8); ARG_P(9),
     p0, i1, p2, p3, i4, i5, i6, i7, i8, p9)
CALL(attn_fwd, 12, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_I(5); ARG_I(6); ARG_I(7); ARG_I(8); ARG_I(9); ARG_I(10); ARG_P(11),
     p0, p1, p2, p3, p4, i5, i6, i7, i8, i9, i10, p11)
CALL(attn_bwd, 17, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_P(5); ARG_P(6); ARG_P(7); ARG_P(8); ARG_P(9); ARG_I(10); ARG_I(11);
     ARG_I(12); ARG_I(13); ARG_I(14); ARG_I(15); ARG_P(16), p0, p1, p2, p3, p4, p5, p6, p7, p8, p9, i10, i11, i12, i13, i14, i15, p16)
CALL(moe_forward, 6, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_P(5), p0, p1, p2, p3, p4, p5)
CALL(moe_decode, 6, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_P(5), p0, p1, p2, p3, p4, p5)
CALL(moe_backward, 11, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_P(5); ARG_P(6); ARG_P(7); ARG_P(8); ARG_F(9); ARG_P(10),
     p0, p1, p2, p3, p4, p5, p6, p7, p8, f9, p10)
CALL(adamw, 13, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_U(4); ARG_F(5); ARG_F(6); ARG_F(7); ARG_F(8); ARG_F(9);
     ARG_F(10); ARG_P(11); ARG_P(12), p0, p1, p2, p3, (size_t)u4, f5, f6, f7, f8, f9, f10, p11, p12)
CALL(step, 29, ARG_P(0); ARG_P(1); ARG_P(2); ARG_P(3); ARG_P(4); ARG_P(5); ARG_P(6); ARG_P(7); ARG_P(8); ARG_P(9); ARG_I(10); ARG_I(11); ARG_I(12);
     ARG_F(13); ARG_F(14); ARG_F(15); ARG_F(16); ARG_F(17); ARG_P(18); ARG_F(19); ARG_F(20); ARG_I(21); ARG_U(22);
     ARG_I(23); ARG_P(24); ARG_I(25); ARG_I(26); ARG_I(27); ARG_P(28),
     p0, p1, p2, p3, p4, p5, p6, p7, p8, p9, i10, i11, i12, f13, f14, f15, f16, f17, p18, f19, f20, i21, u22, i23, p24, i25, i26, i27, p28)
CALL(gnorm, 8, ARG_P(0); ARG_U(1); ARG_P(2); ARG_P(3); ARG_I(4); ARG_I(5); ARG_P(6); ARG_P(7), p0, (size_t)u1, p2, p3, i4, i5, p6, p7)
CALL(dec_step, 2, ARG_P(0); ARG_P(1), p0, p1)
CALL(dec_greedy, 6, ARG_P(0); ARG_P(1); ARG_P(2); ARG_I(3); ARG_I(4); ARG_P(5), p0, p1, p2, i3, i4, p5)

static PyObject *set_error_class(PyObject *self, PyObject *cls)
{
    (void)self;
    Py_INCREF(cls);
    Py_XSETREF(error_class, cls);
    Py_RETURN_NONE;
}

#define ENTRY(NAME) {#NAME, (PyCFunction)(void (*)(void))py_##NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    ENTRY(gemv_decode), ENTRY(linear_fwd), ENTRY(linear_dgrad), ENTRY(linear_wgrad), ENTRY(gemm_nt), ENTRY(embed), ENTRY(rmsnorm_fwd),
    ENTRY(rmsnorm_bwd), ENTRY(rope), ENTRY(attn_fwd), ENTRY(attn_bwd), ENTRY(moe_forward), ENTRY(moe_decode), ENTRY(moe_backward), ENTRY(adamw),
    ENTRY(step), ENTRY(gnorm), ENTRY(dec_step), ENTRY(dec_greedy),
    {"set_error_class", set_error_class, METH_O, NULL},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pycalls", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__pycalls(void)
{
    name_data_ptr = PyUnicode_InternFromString("data_ptr");
    return name_data_ptr ? PyModule_Create(&module) : NULL;
}
