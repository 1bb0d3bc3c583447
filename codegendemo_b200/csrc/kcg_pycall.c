/* The two launches a Python program makes most, as one C call each: tensors to addresses, Python numbers to C ones, the
 * launch, its status back. The same entries of libkcg_b200.so serve them through ctypes; there `launchKernel` took 4.0 us
 * without the driver's part, here it takes 0.9 (the whole of `matmul`, whose contiguous operands also skip the row-pitch
 * questions, 8.7 -> 3.9 on the same host). `bind` is given the entries' addresses, so this module is linked against neither the library nor torch. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#include "../../include/kcg_b200.h"

typedef int (*GemmFn)(uint64_t, const kcg_kernel_info*, int, uint64_t, uint64_t, uint64_t, uint64_t, int64_t, int64_t,
                      int64_t, int, const kcg_epilogue*);
typedef int (*AttentionFn)(int, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, int, int, int, int, int, float);
static GemmFn g_gemm;
static AttentionFn g_attention;
static PyObject* g_data_ptr;

/* int(o) and float(o) of an argument, as C numbers; the exact types first. -1 with an exception set on failure. */
static int u64_of(PyObject* o, uint64_t* out) {
  if (PyLong_Check(o)) {
    *out = PyLong_AsUnsignedLongLong(o);
  } else {
    PyObject* i = PyNumber_Long(o);
    if (!i) return -1;
    *out = PyLong_AsUnsignedLongLong(i);
    Py_DECREF(i);
  }
  return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
}

static int i64_of(PyObject* o, int64_t* out) {
  if (PyLong_Check(o)) {
    *out = PyLong_AsLongLong(o);
  } else {
    PyObject* i = PyNumber_Long(o);
    if (!i) return -1;
    *out = PyLong_AsLongLong(i);
    Py_DECREF(i);
  }
  return *out == -1 && PyErr_Occurred() ? -1 : 0;
}

static int int_of(PyObject* o, int* out) {
  int64_t v;
  if (i64_of(o, &v)) return -1;
  *out = (int)v;
  return 0;
}

static int double_of(PyObject* o, double* out) {
  if (PyFloat_CheckExact(o)) {
    *out = PyFloat_AS_DOUBLE(o);
    return 0;
  }
  PyObject* f = PyNumber_Float(o);
  if (!f) return -1;
  *out = PyFloat_AS_DOUBLE(f);
  Py_DECREF(f);
  return 0;
}

/* Address of an argument: an int, or what its data_ptr() returns. */
static int pointer_of(PyObject* o, uint64_t* out) {
  if (PyLong_Check(o)) return u64_of(o, out);
  if (o == Py_None) {
    PyErr_SetString(PyExc_TypeError, "KCG launcher: pointer argument is None");
    return -1;
  }
  PyObject* r = PyObject_CallMethodNoArgs(o, g_data_ptr);
  if (!r) {
    if (PyErr_ExceptionMatches(PyExc_AttributeError)) {
      PyObject *type, *value, *trace;
      PyErr_Fetch(&type, &value, &trace);
      const int has = PyObject_HasAttr(o, g_data_ptr);  /* then the error came from inside the method */
      PyErr_Restore(type, value, trace);
      if (!has) PyErr_SetString(PyExc_TypeError, "Pointer argument must be either uint64 or have data_ptr method");
    }
    return -1;
  }
  const int e = u64_of(r, out);
  Py_DECREF(r);
  return e;
}

static PyObject* bind(PyObject* self, PyObject* args) {
  unsigned long long gemm, attention;
  if (!PyArg_ParseTuple(args, "KK", &gemm, &attention)) return NULL;
  g_gemm = (GemmFn)(uintptr_t)gemm;
  g_attention = (AttentionFn)(uintptr_t)attention;
  Py_RETURN_NONE;
}

/* gemm(function, info, device, stream, a, b, c, lda, ldb, ldc, batch, alpha, beta, bias, relu) -> status */
static PyObject* gemm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 15 || !g_gemm) {
    PyErr_SetString(PyExc_TypeError, "gemm takes 15 arguments, after bind");
    return NULL;
  }
  uint64_t function, info, stream, p[3];
  int64_t ld[3];
  int device, batch;
  double alpha, beta;
  if (u64_of(a[0], &function) || u64_of(a[1], &info) || int_of(a[2], &device) || u64_of(a[3], &stream)) return NULL;
  for (int i = 0; i < 3; ++i)
    if (pointer_of(a[4 + i], &p[i]) || i64_of(a[7 + i], &ld[i])) return NULL;
  if (int_of(a[10], &batch) || double_of(a[11], &alpha) || double_of(a[12], &beta)) return NULL;
  const int relu = PyObject_IsTrue(a[14]);
  if (relu < 0) return NULL;
  kcg_epilogue epi = {(float)alpha, (float)beta, 0, relu, {0, 0, 0}};
  if (a[13] != Py_None && pointer_of(a[13], &epi.bias)) return NULL;
  const int fused = alpha != 1.0 || beta != 0.0 || a[13] != Py_None || relu;
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_gemm(function, (const kcg_kernel_info*)(uintptr_t)info, device, stream, p[0], p[1], p[2], ld[0], ld[1], ld[2],
                  batch, fused ? &epi : NULL);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

/* attention(device, stream, q, k, v, out, dtype, heads, sq, sk, d, scale) -> status */
static PyObject* attention(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 12 || !g_attention) {
    PyErr_SetString(PyExc_TypeError, "attention takes 12 arguments, after bind");
    return NULL;
  }
  uint64_t stream, p[4];
  int device, v[5];
  double scale;
  if (int_of(a[0], &device) || u64_of(a[1], &stream)) return NULL;
  for (int i = 0; i < 4; ++i)
    if (pointer_of(a[2 + i], &p[i])) return NULL;
  for (int i = 0; i < 5; ++i)
    if (int_of(a[6 + i], &v[i])) return NULL;
  if (double_of(a[11], &scale)) return NULL;
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_attention(device, stream, p[0], p[1], p[2], p[3], v[0], v[1], v[2], v[3], v[4], (float)scale);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

static PyMethodDef g_methods[] = {{"bind", bind, METH_VARARGS, "addresses of the library's entries"},
                                  {"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, "kcg_launch_gemm_strided"},
                                  {"attention", (PyCFunction)(void (*)(void))attention, METH_FASTCALL, "kcg_attention_fwd"},
                                  {NULL, NULL, 0, NULL}};
static struct PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_pycall", NULL, -1, g_methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__pycall(void) {
  g_data_ptr = PyUnicode_InternFromString("data_ptr");
  return g_data_ptr ? PyModule_Create(&g_module) : NULL;
}
