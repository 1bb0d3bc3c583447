// The warm call of the operators in kcg/matmul_op.py, from torch tensors to the queued launch, as one C++ call: shapes, types
// and strides from the tensors themselves, the kernel from a table, the result from torch's allocator, the stream torch's
// current one. It takes only what needs no decision - plain contiguous CUDA tensors of a shape whose kernel the Python
// operator has built and launched before, no mode that watches torch's calls - and answers None to everything else, which
// then goes the operator's own way, with its checks and errors. Host time of a warm call (256 x 1024 x 512, B200 host): `matmul`
// 6.5 us through Python, of them 2.2 the launch and 1.8 the result's allocation, 3.6 here; the GPU needs 4.4. Calls in a row 6.6 -> 4.3.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/version.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <unordered_map>

#include "../../include/kcg_b200.h"

namespace {

using GemmFn = int (*)(uint64_t, const kcg_kernel_info*, int, uint64_t, uint64_t, uint64_t, uint64_t, int64_t, int64_t,
                       int64_t, int, const kcg_epilogue*);
using AttentionFn = int (*)(int, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, int, int, int, int, int, float);
GemmFn g_gemm = nullptr;
AttentionFn g_attention = nullptr;
PyObject* g_check = nullptr;  // raises the error of a status

// torch's allocator asks before it takes memory from the device: the library's workspaces, which it cannot see, are given back
// when memory is low. (No GIL here, and no call of the library comes back to the allocator.)
std::atomic<bool (*)(int)> g_trim{nullptr};
struct GiveBack final : c10::FreeMemoryCallback {
  bool Execute() override {
    bool (*trim)(int) = g_trim.load();
    return trim && trim(c10::cuda::current_device());
  }
};

// What the operator chose a kernel by. Written and read with the GIL held.
struct Shape {
  int64_t m, n, k, batch;  // batch 0: not a batched product
  int32_t dtype, device, b_transposed;
  bool operator==(const Shape& o) const {
    return m == o.m && n == o.n && k == o.k && batch == o.batch && dtype == o.dtype && device == o.device &&
           b_transposed == o.b_transposed;
  }
};
struct ShapeHash {
  size_t operator()(const Shape& s) const {
    uint64_t h = 0;
    for (uint64_t v : {static_cast<uint64_t>(s.m), static_cast<uint64_t>(s.n), static_cast<uint64_t>(s.k),
                       static_cast<uint64_t>(s.batch),
                       static_cast<uint64_t>(s.dtype) << 32 | static_cast<uint64_t>(s.device) << 8 | static_cast<uint64_t>(s.b_transposed)}) {
      h = (h ^ v) * 0x9e3779b97f4a7c15ull;
      h ^= h >> 32;
    }
    return static_cast<size_t>(h);
  }
};
struct Kernel {
  uint64_t function;
  const kcg_kernel_info* info;
  PyObject* owner;  // the launcher that both belong to
};
std::unordered_map<Shape, Kernel, ShapeHash> g_kernels;

// The tensor of an argument this path takes: a plain CUDA tensor that lies in memory as its shape says.
const at::Tensor* plain(PyObject* o, int64_t dim) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.dim() != dim || t.layout() != at::kStrided || !t.has_storage() || !t.is_contiguous()) return nullptr;
  return &t;
}

// 16-bit types and fp32, by the numbers of the configs
int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return KCG_DTYPE_FLOAT16;
    case at::kBFloat16: return KCG_DTYPE_BFLOAT16;
    case at::kFloat: return KCG_DTYPE_FLOAT32;
    default: return 0;
  }
}

// Something that sees or replaces torch's calls is at work: the result has to be made by one of them.
bool watched() { return at::impl::torch_function_mode_enabled() || c10::impl::dispatch_mode_enabled(); }

uint64_t address(const at::Tensor& t) { return reinterpret_cast<uint64_t>(t.const_data_ptr()); }

PyObject* finish(int status, at::Tensor&& result) {
  if (status == 0) return THPVariable_Wrap(std::move(result));
  PyObject* r = PyObject_CallFunction(g_check, "i", status);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "launch failed with status %d", status);
  return nullptr;
}

// Launches the product if its kernel is known; None if it is not.
PyObject* product(const Shape& shape, const at::Tensor& a, const at::Tensor& b, at::IntArrayRef sizes, PyObject* bias,
                  PyObject* relu_arg) {
  const auto it = g_kernels.find(shape);
  if (it == g_kernels.end() || watched()) Py_RETURN_NONE;
  kcg_epilogue epi = {1.f, 0.f, 0, 0, {0, 0, 0}};
  bool fused = false;
  if (relu_arg != Py_False) {
    if (relu_arg != Py_True) Py_RETURN_NONE;
    epi.relu = 1;
    fused = true;
  }
  if (bias != Py_None) {
    const at::Tensor* t = plain(bias, 1);
    if (!t || t->device() != a.device()) Py_RETURN_NONE;
    epi.bias = address(*t);
    fused = true;
  }
  const Kernel kernel = it->second;
  // The launch reads the owner's info with the GIL released, and another thread may put another owner in its place.
  const auto owner = THPObjectPtr(Py_NewRef(kernel.owner));
  const uint64_t stream = reinterpret_cast<uint64_t>(c10::cuda::getCurrentCUDAStream(a.device().index()).stream());
  at::Tensor c = at::detail::empty_cuda(sizes, a.scalar_type(), a.device(), std::nullopt);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_gemm(kernel.function, kernel.info, shape.device, stream, address(a), address(b), reinterpret_cast<uint64_t>(c.mutable_data_ptr()),
                  0, 0, 0, shape.batch > 0 ? static_cast<int>(shape.batch) : 1, fused ? &epi : nullptr);
  Py_END_ALLOW_THREADS
  return finish(status, std::move(c));
}

// matmul(a, b, bias, relu, b_transposed) -> tensor or None
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !g_gemm) Py_RETURN_NONE;
  if (args[4] != Py_False && args[4] != Py_True) Py_RETURN_NONE;
  const at::Tensor *a = plain(args[0], 2), *b = plain(args[1], 2);
  if (!a || !b || a->scalar_type() != b->scalar_type() || a->device() != b->device()) Py_RETURN_NONE;
  const bool bt = args[4] == Py_True;
  const Shape shape{a->size(0), b->size(bt ? 0 : 1), a->size(1), 0, dtype_of(*a), a->device().index(), bt ? 1 : 0};
  if (!shape.dtype || b->size(bt ? 1 : 0) != shape.k) Py_RETURN_NONE;
  return product(shape, *a, *b, {shape.m, shape.n}, args[2], args[3]);
  END_HANDLE_TH_ERRORS
}

// bmm(a, b, bias, relu) -> tensor or None
PyObject* bmm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !g_gemm) Py_RETURN_NONE;
  const at::Tensor *a = plain(args[0], 3), *b = plain(args[1], 3);
  if (!a || !b || a->scalar_type() != b->scalar_type() || a->device() != b->device()) Py_RETURN_NONE;
  const Shape shape{a->size(1), b->size(2), a->size(2), a->size(0), dtype_of(*a), a->device().index(), 0};
  if (!shape.dtype || b->size(0) != shape.batch || b->size(1) != shape.k) Py_RETURN_NONE;
  return product(shape, *a, *b, {shape.batch, shape.m, shape.n}, args[2], args[3]);
  END_HANDLE_TH_ERRORS
}

// attention(q, k, v) -> tensor or None; the scale is 1 / sqrt(head dimension)
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || !g_attention) Py_RETURN_NONE;
  const at::Tensor *q = plain(args[0], 3), *k = plain(args[1], 3), *v = plain(args[2], 3);
  if (!q || !k || !v || k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() ||
      k->device() != q->device() || v->device() != q->device() || k->sizes() != v->sizes())
    Py_RETURN_NONE;
  const int64_t heads = q->size(0), sq = q->size(1), d = q->size(2), sk = k->size(1);
  const int dtype = dtype_of(*q);
  if (k->size(0) != heads || k->size(2) != d || (dtype != KCG_DTYPE_FLOAT16 && dtype != KCG_DTYPE_BFLOAT16) ||
      heads > INT32_MAX || sq > INT32_MAX || sk > INT32_MAX || (d != 64 && d != 128) || watched())
    Py_RETURN_NONE;
  const int device = q->device().index();
  const uint64_t stream = reinterpret_cast<uint64_t>(c10::cuda::getCurrentCUDAStream(q->device().index()).stream());
  at::Tensor o = at::detail::empty_cuda(q->sizes(), q->scalar_type(), q->device(), std::nullopt);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_attention(device, stream, address(*q), address(*k), address(*v), reinterpret_cast<uint64_t>(o.mutable_data_ptr()), dtype,
                       static_cast<int>(heads), static_cast<int>(sq), static_cast<int>(sk), static_cast<int>(d),
                       static_cast<float>(1.0 / std::sqrt(static_cast<double>(d))));
  Py_END_ALLOW_THREADS
  return finish(status, std::move(o));
  END_HANDLE_TH_ERRORS
}

// remember(m, n, k, batch, dtype, device, b_transposed, function, info, owner)
PyObject* remember(PyObject*, PyObject* args) {
  Shape s{};
  unsigned long long function, info;
  PyObject* owner;
  long long m, n, k, batch;
  if (!PyArg_ParseTuple(args, "LLLLiiiKKO", &m, &n, &k, &batch, &s.dtype, &s.device, &s.b_transposed, &function, &info, &owner))
    return nullptr;
  s.m = m, s.n = n, s.k = k, s.batch = batch;
  Py_INCREF(owner);
  Kernel& e = g_kernels[s];
  PyObject* old = e.owner;
  e = Kernel{function, reinterpret_cast<const kcg_kernel_info*>(static_cast<uintptr_t>(info)), owner};
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

// bind(kcg_launch_gemm_strided, kcg_attention_fwd, check): addresses and the function that raises a status
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long gemm, attention;
  PyObject* check;
  if (!PyArg_ParseTuple(args, "KKO", &gemm, &attention, &check)) return nullptr;
  Py_INCREF(check);
  Py_XDECREF(g_check);
  g_check = check;
  g_gemm = reinterpret_cast<GemmFn>(static_cast<uintptr_t>(gemm));
  g_attention = reinterpret_cast<AttentionFn>(static_cast<uintptr_t>(attention));
  Py_RETURN_NONE;
}

// bind_trim(kcg_internal_trim_if_low)
PyObject* bind_trim(PyObject*, PyObject* args) {
  unsigned long long trim;
  if (!PyArg_ParseTuple(args, "K", &trim)) return nullptr;
  g_trim = reinterpret_cast<bool (*)(int)>(static_cast<uintptr_t>(trim));
  Py_RETURN_NONE;
}

template <typename F>
PyCFunction fast(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}
PyMethodDef g_methods[] = {{"bind", bind, METH_VARARGS, "addresses of the library's entries"},
                           {"bind_trim", bind_trim, METH_VARARGS, "address of the function that gives memory back"},
                           {"remember", remember, METH_VARARGS, "a shape's kernel"},
                           {"matmul", fast(matmul), METH_FASTCALL, "a product whose kernel is known, or None"},
                           {"bmm", fast(bmm), METH_FASTCALL, "a batched one"},
                           {"attention", fast(attention), METH_FASTCALL, "fused attention, or None"},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torchcall", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

namespace c10 {
REGISTER_FREE_MEMORY_CALLBACK("kcg_workspaces", GiveBack)
}

PyMODINIT_FUNC PyInit__torchcall() {
  PyObject* m = PyModule_Create(&g_module);
  if (m && PyModule_AddStringConstant(m, "TORCH_VERSION", TORCH_VERSION) < 0) Py_CLEAR(m);  // that it was built against
  return m;
}
