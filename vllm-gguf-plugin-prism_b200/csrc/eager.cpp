// The functions of an eager call: plain Python functions over the C-ABI of libgguf_b200, the same bodies as the registered
// operators (op_calls.h).  A decode GEMV runs for 3 to 8 us on the device, and the dispatcher with its boxed arguments
// costs more host time than that per call (a 3072 x 1024 matrix, one token: 12.6 us per call through two registered
// operators, of which the kernel is 3.3).  They answer None whenever the tensors are not plain CUDA tensors (tracing, fake
// tensors, dispatch modes), and the caller then takes the registered operator.
//
// They take tensors apart that Python holds, with torch's own C++ interface, so this module is tied to one Python and to
// the torch it was built against; it refuses to load next to another one, and calls then go through the operators
// (native.py).
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/headeronly/version.h>

#include "op_calls.h"

using at::ScalarType;
using at::Tensor;

namespace {

struct Eager {
  using Tensor = at::Tensor;
  using Guard = c10::cuda::CUDAGuard;
  static c10::DeviceIndex device(const Tensor& t) { return t.get_device(); }
  static void* stream(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(device(t)).stream(); }
  static Tensor empty(const Tensor& like, at::IntArrayRef sizes, ScalarType t) { return at::detail::empty_cuda(sizes, t, like.device(), std::nullopt); }
  static bool has_room(const Tensor& t, int64_t bytes) { return (int64_t)t.storage().nbytes() - t.storage_offset() >= bytes; }
  static Tensor block(const Tensor& t, int64_t row, int64_t rows, int64_t col, int64_t cols) { return t.narrow(0, row, rows).narrow(1, col, cols); }
  static Tensor packed(const Tensor& t) { return t.contiguous(); }
  static void copy(Tensor to, const Tensor& from) { to.copy_(from); }
  // scratch memory of one call, given back to the stream's pool when the call returns
  struct Scratch {
    c10::DataPtr p;
    Scratch(const Tensor&, int64_t bytes) : p(c10::cuda::CUDACachingAllocator::get()->allocate((size_t)(bytes > 0 ? bytes : 1))) {}
    void* get() const { return p.get(); }
  };
};
using Op = gguf_ops::Calls<Eager>;

// Allocation and launches run without the GIL, as an operator's do: cudaMalloc takes a lock and may wait for the device, and
// a launch waits as soon as a thousand are queued (a thread that launches into a full queue held all others for the 0.6 s it
// took to drain).  What is used meanwhile belongs to this call: handles of the tensors, taken while the GIL was held.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <class F> Tensor without_gil(F&& body) {
  Tensor out;
  {
    const NoGil release;
    out = body();
  }
  return out;
}

// Nothing between Python and the kernel wants to see the call: no tracing, functionalization or
// dispatch mode, no tensor subclass.
bool modes_off() {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  const auto inc = c10::impl::tls_local_dispatch_key_set().included_;
  return !inc.has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchDynamicLayerFrontMode}));
}
const Tensor* plain_cuda(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda()) return nullptr;
  const c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::Functionalize,
                                 c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
  return t.key_set().has_any(odd) ? nullptr : &t;
}

// mul_mat(W, X, type, row, op): the three dense products
PyObject* py_mul_mat(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 5, "mul_mat takes 5 arguments");
  const Tensor *W = plain_cuda(a[0]), *X = plain_cuda(a[1]);
  if (!W || !X || !modes_off()) Py_RETURN_NONE;
  const long type = PyLong_AsLong(a[2]), row = PyLong_AsLong(a[3]), op = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  TORCH_CHECK(op == GGUF_B200_OP_GEMV || op == GGUF_B200_OP_MMQ || op == GGUF_B200_OP_DEQUANT_MATMUL, "mul_mat: unknown op");
  static const char* const names[] = {"ggml_mul_mat_vec_a8", "ggml_mul_mat_a8", "", "", "dequant_matmul"};
  const Tensor w = *W, x = *X;
  return THPVariable_Wrap(without_gil([&] { return Op::mul_mat(w, x, type, row, (int)op, names[op], false); }));
  END_HANDLE_TH_ERRORS
}

// embed(ids, W, type, hidden, dtype): the embedding look-up, result shaped [*ids.shape, hidden]
PyObject* py_embed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 5, "embed takes 5 arguments");
  const Tensor *ids = plain_cuda(a[0]), *W = plain_cuda(a[1]);
  if (!ids || !W || !modes_off() || ids->scalar_type() != ScalarType::Long || !ids->is_contiguous() || W->dim() != 2) Py_RETURN_NONE;
  const long type = PyLong_AsLong(a[2]), hidden = PyLong_AsLong(a[3]);
  if (PyErr_Occurred()) return nullptr;
  const ScalarType dt = THPDtype_Check(a[4]) ? reinterpret_cast<THPDtype*>(a[4])->scalar_type : ScalarType::Half;
  const int64_t K = Op::check_weight(*W, type, "embed");
  if (K != hidden || K % 256 != 0 || ids->device() != W->device()) Py_RETURN_NONE;
  const int code = gguf_ops::dtype_code(dt, "embed");
  c10::SmallVector<int64_t, 4> shape(ids->sizes().begin(), ids->sizes().end());
  shape.push_back(hidden);
  const Tensor w = *W, rows = *ids;
  return THPVariable_Wrap(without_gil([&] {
    const Eager::Guard guard(Eager::device(w));
    Tensor out = Eager::empty(w, shape, dt);
    Op::rows_into(w, rows, type, K, out, code);
    return out;
  }));
  END_HANDLE_TH_ERRORS
}

// linear(x, W, type): one layer's product, routed as the dispatcher routes it
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 3, "linear takes 3 arguments");
  const Tensor *X = plain_cuda(a[0]), *W = plain_cuda(a[1]);
  if (!W || !X || X->dim() != 2 || W->dim() != 2 || X->size(0) == 0 || !modes_off()) Py_RETURN_NONE;
  const long type = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  if (gguf_b200_type_size((int)type) == 0) Py_RETURN_NONE;
  const int64_t N = W->size(0);
  const int op = gguf_ops::linear_op(type, X->size(0), N, X->scalar_type());
  if (op < 0) Py_RETURN_NONE;
  const Tensor w = *W, x = *X;
  return THPVariable_Wrap(without_gil([&] { return Op::mul_mat(w, x, type, N, op, "linear", true); }));
  END_HANDLE_TH_ERRORS
}

// linear_runs(x, W, runs): Op::linear_runs with the runs in a tuple
PyObject* py_linear_runs(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 3 && PyTuple_Check(a[2]) && PyTuple_GET_SIZE(a[2]) % 5 == 0, "linear_runs takes x, W and a tuple of runs");
  const Tensor *X = plain_cuda(a[0]), *W = plain_cuda(a[1]);
  if (!W || !X || X->dim() != 2 || X->size(0) == 0 || !modes_off()) Py_RETURN_NONE;
  c10::SmallVector<int64_t, 15> runs(PyTuple_GET_SIZE(a[2]));
  for (size_t i = 0; i < runs.size(); ++i) runs[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(a[2], i));
  if (PyErr_Occurred()) return nullptr;
  for (size_t i = 0; i < runs.size(); i += 5)
    if (gguf_b200_type_size((int)runs[i]) == 0 || gguf_ops::linear_op(runs[i], X->size(0), runs[i + 4], X->scalar_type()) < 0) Py_RETURN_NONE;
  const Tensor w = *W, x = *X;
  return THPVariable_Wrap(without_gil([&] { return Op::linear_runs(x, w, runs.data(), runs.size()); }));
  END_HANDLE_TH_ERRORS
}

// moe(x, W13, W2, topk_weights, topk_ids, type13, type2, act): the whole expert step
PyObject* py_moe(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "moe takes 8 arguments");
  Tensor t[5];
  for (int i = 0; i < 5; ++i) {
    const Tensor* p = plain_cuda(a[i]);
    if (!p) Py_RETURN_NONE;
    t[i] = *p;
  }
  if (!modes_off()) Py_RETURN_NONE;
  const long type13 = PyLong_AsLong(a[5]), type2 = PyLong_AsLong(a[6]), act = PyLong_AsLong(a[7]);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(without_gil([&] { return Op::fused_moe(t[0], t[1], t[2], t[3], t[4], type13, type2, act); }));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"moe", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_moe)), METH_FASTCALL, nullptr},
    {"mul_mat", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_mul_mat)), METH_FASTCALL, nullptr},
    {"embed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_embed)), METH_FASTCALL, nullptr},
    {"linear_runs", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_linear_runs)), METH_FASTCALL, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&py_linear)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_eager", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyObject* PyInit__eager(void) {
  // (the file's name says which Python; the symbols alone do not say which torch)
  PyObject* torch = PyImport_ImportModule("torch");
  if (!torch) return nullptr;
  PyObject* version = PyObject_GetAttrString(torch, "__version__");
  Py_DECREF(torch);
  if (!version) return nullptr;
  PyObject* text = PyObject_Str(version);
  Py_DECREF(version);
  const char* have = text ? PyUnicode_AsUTF8(text) : nullptr;
  if (!have) {
    Py_XDECREF(text);
    return nullptr;
  }
  const std::string built = TORCH_VERSION, run = std::string(have).substr(0, std::string(have).find('+'));
  Py_DECREF(text);
  if (run != built) {
    PyErr_Format(PyExc_ImportError, "built for torch %s, this is %s", built.c_str(), run.c_str());
    return nullptr;
  }
  return PyModule_Create(&module_def);
}
