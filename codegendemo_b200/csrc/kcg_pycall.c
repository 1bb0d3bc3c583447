/* The two launches a Python program makes most, as one C call each: tensors to addresses, Python numbers to C ones, the
 * launch, its status back. The same entries of libkcg_b200.so serve them through ctypes; converting a launch's twelve
 * arguments there took 2.2 us on a host where this takes 0.4 (the whole of `matmul` 9.3 -> 4.9 us, without the driver's
 * part). `bind` is given the entries' addresses, so this module is linked against neither the library nor torch. */
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

/* Address of an argument: an int, or anything with data_ptr(). */
static int pointer_of(PyObject* o, uint64_t* out) {
  if (PyLong_Check(o)) {
    *out = PyLong_AsUnsignedLongLong(o);
    return PyErr_Occurred() ? -1 : 0;
  }
  if (o == Py_None) {
    PyErr_SetString(PyExc_TypeError, "KCG launcher: pointer argument is None");
    return -1;
  }
  PyObject* r = PyObject_CallMethodNoArgs(o, g_data_ptr);
  if (!r) {
    if (PyErr_ExceptionMatches(PyExc_AttributeError))
      PyErr_SetString(PyExc_TypeError, "Pointer argument must be either uint64 or have data_ptr method");
    return -1;
  }
  *out = PyLong_AsUnsignedLongLong(r);
  Py_DECREF(r);
  return PyErr_Occurred() ? -1 : 0;
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
  const uint64_t function = PyLong_AsUnsignedLongLong(a[0]), info = PyLong_AsUnsignedLongLong(a[1]);
  const int device = (int)PyLong_AsLong(a[2]);
  const uint64_t stream = PyLong_AsUnsignedLongLong(a[3]);
  if (PyErr_Occurred()) return NULL;
  uint64_t p[3];
  for (int i = 0; i < 3; ++i)
    if (pointer_of(a[4 + i], &p[i])) return NULL;
  const int64_t lda = PyLong_AsLongLong(a[7]), ldb = PyLong_AsLongLong(a[8]), ldc = PyLong_AsLongLong(a[9]);
  const int batch = (int)PyLong_AsLong(a[10]);
  const double alpha = PyFloat_AsDouble(a[11]), beta = PyFloat_AsDouble(a[12]);
  const int relu = PyObject_IsTrue(a[14]);
  if (PyErr_Occurred()) return NULL;
  kcg_epilogue epi = {(float)alpha, (float)beta, 0, relu, {0, 0, 0}};
  if (a[13] != Py_None && pointer_of(a[13], &epi.bias)) return NULL;
  const int fused = alpha != 1.0 || beta != 0.0 || a[13] != Py_None || relu;
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_gemm(function, (const kcg_kernel_info*)(uintptr_t)info, device, stream, p[0], p[1], p[2], lda, ldb, ldc, batch,
                  fused ? &epi : NULL);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(status);
}

/* attention(device, stream, q, k, v, out, dtype, heads, sq, sk, d, scale) -> status */
static PyObject* attention(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 12 || !g_attention) {
    PyErr_SetString(PyExc_TypeError, "attention takes 12 arguments, after bind");
    return NULL;
  }
  uint64_t p[4];
  for (int i = 0; i < 4; ++i)
    if (pointer_of(a[2 + i], &p[i])) return NULL;
  const uint64_t stream = PyLong_AsUnsignedLongLong(a[1]);
  const long v[6] = {PyLong_AsLong(a[0]), PyLong_AsLong(a[6]), PyLong_AsLong(a[7]),
                     PyLong_AsLong(a[8]), PyLong_AsLong(a[9]), PyLong_AsLong(a[10])};
  const double scale = PyFloat_AsDouble(a[11]);
  if (PyErr_Occurred()) return NULL;
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_attention((int)v[0], stream, p[0], p[1], p[2], p[3], (int)v[1], (int)v[2], (int)v[3], (int)v[4], (int)v[5],
                       (float)scale);
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
