/*
 * CPython binding of the entry points that a program calls once per layer and
 * step.  A call through ctypes costs 1.5 us of interpreter time (argument
 * conversion, the address of each tensor, the wrapper itself) next to the 1.9 us
 * the driver takes for a launch, which is what bounds a small layer; here it costs
 * about a quarter of that.  The functions take the values of the ctypes layer (a
 * context handle as int, ctypes structures, anything with an address) and return
 * the status code; capi.py raises on it.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "poplibs_b200.h"

static PyObject *s_data_ptr, *s_ctypes, *s_data;
/* ctypes.ArgumentError and the structures of the ctypes layer (set_types) */
static PyObject *t_error, *t_matmul_desc, *t_conv_params, *t_conv_options;

/* A value of the wrong type raises what ctypes raises for it. */
static int argument_error(PyObject *o, const char *expected) {
  if (PyErr_ExceptionMatches(PyExc_TypeError)) {
    PyErr_Clear();
    PyErr_Format(t_error ? t_error : PyExc_TypeError, "expected %s instead of %s", expected, Py_TYPE(o)->tp_name);
  }
  return -1;
}

/* Device or host address of None, an int, a torch tensor or a numpy array. */
static int address(PyObject *o, void **out) {
  if (o == Py_None) {
    *out = NULL;
    return 0;
  }
  PyObject *v = NULL;
  if (PyLong_Check(o)) {
    Py_INCREF(o);
    v = o;
  } else {
    PyObject *method = PyObject_GetAttr(o, s_data_ptr);
    if (method != NULL) {
      v = PyObject_CallNoArgs(method);
      Py_DECREF(method);
    } else {
      if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return -1;
      PyErr_Clear();
      PyObject *c = PyObject_GetAttr(o, s_ctypes);
      if (c == NULL) {
        PyErr_Format(PyExc_TypeError, "cannot take the address of %R", (PyObject *)Py_TYPE(o));
        return -1;
      }
      v = PyObject_GetAttr(c, s_data);
      Py_DECREF(c);
    }
    if (v == NULL) return -1;
  }
  *out = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  return *out == NULL && PyErr_Occurred() ? -1 : 0;
}

/* Address of a ctypes structure of type `type` (None: NULL, where it may be left
 * out).  The caller's reference keeps it alive for the call. */
static int structure(PyObject *o, PyObject *type, int optional, const void **out) {
  Py_buffer b;
  if (optional && o == Py_None) {
    *out = NULL;
    return 0;
  }
  if (type == NULL || !PyObject_TypeCheck(o, (PyTypeObject *)type)) {
    PyErr_Format(t_error ? t_error : PyExc_TypeError, "expected %s instead of %s",
                 type ? ((PyTypeObject *)type)->tp_name : "a structure", Py_TYPE(o)->tp_name);
    return -1;
  }
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) return -1;
  *out = b.buf;
  PyBuffer_Release(&b);
  return 0;
}

static int as_float(PyObject *o, float *out) {
  const double v = PyFloat_AsDouble(o);
  *out = (float)v;
  return v == -1.0 && PyErr_Occurred() ? argument_error(o, "a number") : 0;
}
/* An integer of at most `most`: what does not fit is an error, not cut off. */
static int as_unsigned(PyObject *o, uint64_t most, uint64_t *out) {
  PyObject *v = PyNumber_Index(o);
  if (v == NULL) return argument_error(o, "an integer");
  *out = PyLong_AsUnsignedLongLong(v);
  Py_DECREF(v);
  if (*out == (uint64_t)-1 && PyErr_Occurred()) return -1;
  if (*out <= most) return 0;
  PyErr_Format(PyExc_OverflowError, "%R does not fit the argument's type", o);
  return -1;
}
static int as_int(PyObject *o, int *out) {
  const long v = PyLong_AsLong(o);
  *out = (int)v;
  if (v == -1 && PyErr_Occurred()) return argument_error(o, "an integer");
  if (v == *out) return 0;
  PyErr_Format(PyExc_OverflowError, "%R does not fit the argument's type", o);
  return -1;
}

#define FUNCTION(name) static PyObject *name(PyObject *self, PyObject *const *a, Py_ssize_t n)
#define ARGS(count)                                                                     \
  (void)self;                                                                           \
  if (n != (count)) return PyErr_Format(PyExc_TypeError, "%d arguments expected", (count))
#define CONTEXT(i)                                                       \
  plb_context *ctx = (plb_context *)PyLong_AsVoidPtr(a[i]);              \
  if (ctx == NULL && PyErr_Occurred()) return NULL
#define PTR(i, p)         \
  void *p;                \
  if (address(a[i], &p)) return NULL
#define STRUCT(i, type, py_type, optional, p)                         \
  const void *p##_v;                                                  \
  if (structure(a[i], py_type, optional, &p##_v)) return NULL;        \
  const type *p = (const type *)p##_v
#define INT(i, v) \
  int v;          \
  if (as_int(a[i], &v)) return NULL
#define U64(i, v) \
  uint64_t v;     \
  if (as_unsigned(a[i], UINT64_MAX, &v)) return NULL
#define U32(i, v)    \
  uint64_t v##_wide; \
  if (as_unsigned(a[i], UINT32_MAX, &v##_wide)) return NULL; \
  const uint32_t v = (uint32_t)v##_wide
#define FLOAT(i, v) \
  float v;          \
  if (as_float(a[i], &v)) return NULL
#define CALL(expr)         \
  int rc;                  \
  Py_BEGIN_ALLOW_THREADS   \
  rc = (expr);             \
  Py_END_ALLOW_THREADS     \
  return PyLong_FromLong(rc)

FUNCTION(matmul) {
  ARGS(6);
  CONTEXT(0);
  STRUCT(1, plb_matmul_desc, t_matmul_desc, 0, d);
  PTR(2, pa);
  PTR(3, pb);
  PTR(4, pc);
  PTR(5, pd);
  CALL(plb_matmul(ctx, d, pa, pb, pc, pd));
}
FUNCTION(convolution) {
  ARGS(8);
  CONTEXT(0);
  STRUCT(1, plb_conv_params, t_conv_params, 0, p);
  STRUCT(2, plb_conv_options, t_conv_options, 1, o);
  PTR(3, x);
  PTR(4, w);
  PTR(5, bias);
  PTR(6, out);
  INT(7, flip);
  CALL(plb_convolution(ctx, p, o, x, w, (const float *)bias, out, flip));
}
FUNCTION(conv_bwd) {
  ARGS(6);
  CONTEXT(0);
  STRUCT(1, plb_conv_params, t_conv_params, 0, p);
  STRUCT(2, plb_conv_options, t_conv_options, 1, o);
  PTR(3, dy);
  PTR(4, w);
  PTR(5, dx);
  CALL(plb_conv_bwd(ctx, p, o, dy, w, dx));
}
FUNCTION(conv_wu) {
  ARGS(7);
  CONTEXT(0);
  STRUCT(1, plb_conv_params, t_conv_params, 0, p);
  STRUCT(2, plb_conv_options, t_conv_options, 1, o);
  PTR(3, x);
  PTR(4, dy);
  PTR(5, dw);
  PTR(6, dw32);
  CALL(plb_conv_wu(ctx, p, o, x, dy, dw, (float *)dw32));
}
FUNCTION(scaled_add_to) {
  ARGS(6);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, w);
  PTR(3, d);
  FLOAT(4, scale);
  U64(5, count);
  CALL(plb_scaled_add_to(ctx, dtype, w, (const float *)d, scale, (size_t)count));
}
FUNCTION(cast_from_f32) {
  ARGS(5);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, dst);
  PTR(3, src);
  U64(4, count);
  CALL(plb_cast_from_f32(ctx, dtype, dst, (const float *)src, (size_t)count));
}
FUNCTION(conv_bias_update) {
  ARGS(8);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, dy);
  U64(3, pixels);
  U32(4, chans);
  INT(5, bias_dtype);
  PTR(6, bias);
  FLOAT(7, scale);
  CALL(plb_conv_bias_update(ctx, dtype, dy, pixels, chans, bias_dtype, bias, scale));
}
FUNCTION(norm_moments) {
  ARGS(9);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, x);
  U64(3, pixels);
  U32(4, chans);
  FLOAT(5, scale);
  PTR(6, centre);
  PTR(7, mean);
  PTR(8, power);
  CALL(plb_norm_moments(ctx, dtype, x, pixels, chans, scale, centre, mean, (float *)power));
}
FUNCTION(norm_statistics) {
  ARGS(10);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, x);
  U64(3, pixels);
  U32(4, chans);
  FLOAT(5, eps);
  FLOAT(6, scale_var);
  PTR(7, mean);
  PTR(8, inv_std);
  PTR(9, power);
  CALL(plb_norm_statistics(ctx, dtype, x, pixels, chans, eps, scale_var, mean, inv_std, (float *)power));
}
FUNCTION(norm_normalise) {
  ARGS(11);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, x);
  PTR(3, mean);
  PTR(4, inv_std);
  PTR(5, gamma);
  PTR(6, beta);
  U64(7, pixels);
  U32(8, chans);
  PTR(9, whitened);
  PTR(10, out);
  CALL(plb_norm_normalise(ctx, dtype, x, mean, inv_std, gamma, beta, pixels, chans, whitened, out));
}
FUNCTION(norm_whiten) {
  ARGS(8);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, x);
  PTR(3, mean);
  PTR(4, inv_std);
  U64(5, pixels);
  U32(6, chans);
  PTR(7, out);
  CALL(plb_norm_whiten(ctx, dtype, x, mean, inv_std, pixels, chans, out));
}
FUNCTION(norm_scale_shift) {
  ARGS(8);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, x);
  PTR(3, scale);
  PTR(4, shift);
  U64(5, pixels);
  U32(6, chans);
  PTR(7, out);
  CALL(plb_norm_scale_shift(ctx, dtype, x, scale, shift, pixels, chans, out));
}
FUNCTION(norm_param_gradients) {
  ARGS(11);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, whitened);
  PTR(3, grads);
  U64(4, pixels);
  U32(5, chans);
  FLOAT(6, scale);
  PTR(7, gamma);
  PTR(8, beta);
  PTR(9, gamma32);
  PTR(10, beta32);
  CALL(plb_norm_param_gradients(ctx, dtype, whitened, grads, pixels, chans, scale, gamma, beta,
                                (float *)gamma32, (float *)beta32));
}
FUNCTION(norm_statistics_gradients) {
  ARGS(10);
  CONTEXT(0);
  INT(1, dtype);
  PTR(2, whitened);
  PTR(3, grads);
  PTR(4, inv_std);
  PTR(5, var_delta);
  PTR(6, mean_delta);
  U64(7, pixels);
  U32(8, chans);
  PTR(9, out);
  CALL(plb_norm_statistics_gradients(ctx, dtype, whitened, grads, inv_std, var_delta, mean_delta, pixels,
                                     chans, out));
}

/* ctypes.ArgumentError, MatmulDesc, ConvParams, ConvOptions: once, by capi.py. */
FUNCTION(set_types) {
  ARGS(4);
  PyObject **const to[] = {&t_error, &t_matmul_desc, &t_conv_params, &t_conv_options};
  for (int i = 0; i < 4; ++i) {
    if (!PyType_Check(a[i])) return PyErr_Format(PyExc_TypeError, "types expected");
    Py_INCREF(a[i]);
    PyObject *old = *to[i];
    *to[i] = a[i];
    Py_XDECREF(old);
  }
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    METHOD(matmul),         METHOD(convolution),    METHOD(conv_bwd),
    METHOD(conv_wu),        METHOD(scaled_add_to),  METHOD(cast_from_f32),
    METHOD(conv_bias_update), METHOD(norm_moments), METHOD(norm_statistics),
    METHOD(norm_normalise), METHOD(norm_whiten),    METHOD(norm_scale_shift),
    METHOD(norm_param_gradients), METHOD(norm_statistics_gradients), METHOD(set_types),
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__binding(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_ctypes = PyUnicode_InternFromString("ctypes");
  s_data = PyUnicode_InternFromString("data");
  if (s_data_ptr == NULL || s_ctypes == NULL || s_data == NULL) return NULL;
  return PyModule_Create(&module);
}
