// Torch library `_C_gguf` over the C-ABI of libgguf_b200: the six operator schemas of the
// reference's binding file (vllm_gguf_plugin/csrc/torch_bindings.cpp:22-53), registered on the
// same keys (ops on CUDA, ggml_moe_get_block_size as CompositeExplicitAutograd), so
// `vllm_gguf_plugin.ops` finds `torch.ops._C_gguf.*` unchanged.  This file only validates tensors,
// allocates the output and the scratch memory from torch's caching allocator (so CUDA-graph
// capture works as in the reference), resolves the current stream and turns error codes into
// exceptions.  All arithmetic lives behind gguf_b200.h.
//
// The same functions are also plain Python functions of this module (mul_mat, linear, embed, moe):
// what an eager call goes through.  A decode GEMV runs for 3 to 8 us on the device, and the
// dispatcher with its boxed arguments costs more host time than that per call (a 3072 x 1024
// matrix, one token: 12.6 us per call through two registered operators, of which the kernel is
// 3.3).  They answer None whenever the tensors are not plain CUDA tensors (tracing, fake tensors,
// dispatch modes), and the caller then takes the registered operator.
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
#include <torch/library.h>

#include <optional>
#include <string>

#include "../../include/gguf_b200.h"

using at::ScalarType;
using at::Tensor;

namespace {

void* current_stream(c10::DeviceIndex dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }

int dtype_code(ScalarType t, const char* what) {
  switch (t) {
    case ScalarType::Float: return GGUF_B200_F32;
    case ScalarType::Half: return GGUF_B200_F16;
    case ScalarType::BFloat16: return GGUF_B200_BF16;
    default: break;
  }
  TORCH_CHECK(false, what, ": expected a float32, float16 or bfloat16 tensor");
}

void check_rc(int rc, const char* op) { TORCH_CHECK(rc == GGUF_B200_OK, op, " failed: ", gguf_b200_error_string(rc)); }

// Weights are raw GGUF bytes: uint8, contiguous, last dim a whole number of blocks.
int64_t check_weight(const Tensor& W, int64_t type, const char* op) {
  const int ts = gguf_b200_type_size((int)type);
  TORCH_CHECK(ts > 0, op, ": unsupported GGML quantization type ", std::to_string(type));
  TORCH_CHECK(W.scalar_type() == ScalarType::Byte, op, ": W must be a uint8 tensor of raw GGUF blocks");
  TORCH_CHECK(W.is_contiguous(), op, ": W must be contiguous");
  TORCH_CHECK(W.dim() >= 1 && W.size(-1) % ts == 0, op, ": last dim of W is not a whole number of blocks");
  return W.size(-1) / ts * gguf_b200_block_size((int)type);  // K
}

Tensor new_tensor(at::IntArrayRef sizes, ScalarType t, c10::Device dev) { return at::detail::empty_cuda(sizes, t, dev, std::nullopt); }

// scratch memory of one call, given back to the stream's pool when the call returns
struct Scratch {
  c10::DataPtr p;
  explicit Scratch(int64_t bytes) : p(c10::cuda::CUDACachingAllocator::get()->allocate((size_t)(bytes > 0 ? bytes : 1))) {}
  void* get() const { return p.get(); }
};

}  // namespace

Tensor ggml_dequantize(const Tensor& W, int64_t type, int64_t m, int64_t n, std::optional<ScalarType> dtype) {
  const c10::cuda::CUDAGuard guard(W.device());
  check_weight(W, type, "ggml_dequantize");
  const ScalarType dt = dtype.value_or(ScalarType::Half);
  const int code = dtype_code(dt, "ggml_dequantize");
  const int ts = gguf_b200_type_size((int)type), bs = gguf_b200_block_size((int)type);
  TORCH_CHECK(m >= 0 && n >= 0 && (m * n) % bs == 0, "ggml_dequantize: m*n must be a multiple of the block size");
  TORCH_CHECK(W.numel() >= m * n / bs * ts, "ggml_dequantize: W holds fewer than m*n values");
  Tensor out = new_tensor({m, n}, dt, W.device());  // every element is written by the kernel
  check_rc(gguf_b200_dequantize(W.data_ptr(), (int)type, out.data_ptr(), code, m * n, current_stream(W.get_device())), "ggml_dequantize");
  return out;
}

// rows `ids` (contiguous int64, any shape) of the packed weight into `out`
static void rows_into(const Tensor& W, const Tensor& ids, int64_t type, int64_t K, const Tensor& out, int code) {
  check_rc(gguf_b200_dequantize_rows(W.data_ptr(), (int)type, static_cast<const int64_t*>(ids.data_ptr()), ids.numel(), K, W.size(0),
                                     out.data_ptr(), code, current_stream(W.get_device())),
           "dequantize_rows");
}

// Embedding look-up: rows `ids` of the packed weight, dequantized (replaces index_select +
// ggml_dequantize of the reference's embedding caller, quantization/vocal_embeds.py:88-96).
Tensor dequantize_rows(const Tensor& W, const Tensor& ids, int64_t type, std::optional<ScalarType> dtype) {
  const c10::cuda::CUDAGuard guard(W.device());
  const int64_t K = check_weight(W, type, "dequantize_rows");
  TORCH_CHECK(W.dim() == 2, "dequantize_rows: W must be [rows, bytes]");
  TORCH_CHECK(ids.scalar_type() == ScalarType::Long && ids.is_contiguous() && ids.dim() == 1,
              "dequantize_rows: ids must be a contiguous 1-D int64 tensor");
  TORCH_CHECK(K % 256 == 0, "dequantize_rows: the row length must be a multiple of 256");
  const ScalarType dt = dtype.value_or(ScalarType::Half);
  const int code = dtype_code(dt, "dequantize_rows");
  Tensor out = new_tensor({ids.size(0), K}, dt, W.device());
  rows_into(W, ids, type, K, out, code);
  return out;
}

static Tensor matmul_common(const Tensor& W, const Tensor& X, int64_t type, int64_t row, int op, const char* name) {
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t K = check_weight(W, type, name);
  TORCH_CHECK(X.dim() == 2 && X.is_contiguous(), name, ": X must be a contiguous [tokens, K] tensor");
  TORCH_CHECK(X.size(1) == K, name, ": X.shape[1] does not match the K implied by W");
  TORCH_CHECK(row >= 0 && W.numel() / W.size(-1) >= row, name, ": W has fewer than `row` rows");
  const int code = dtype_code(X.scalar_type(), name);
  const int64_t M = X.size(0);
  Tensor Y = new_tensor({M, row}, X.scalar_type(), X.device());
  if (M == 0 || row == 0) return Y;
  const int64_t ws_bytes = gguf_b200_scratch_bytes(op, (int)type, M, row, K);
  const Scratch ws(ws_bytes);
  void* s = current_stream(X.get_device());
  int rc;
  if (op == GGUF_B200_OP_GEMV)
    rc = gguf_b200_mul_mat_vec_a8(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
  else if (op == GGUF_B200_OP_MMQ)
    rc = gguf_b200_mul_mat_a8(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
  else
    rc = gguf_b200_dequant_matmul(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
  check_rc(rc, name);
  return Y;
}

Tensor ggml_mul_mat_vec_a8(const Tensor& W, const Tensor& X, int64_t type, int64_t row) {
  return matmul_common(W, X, type, row, GGUF_B200_OP_GEMV, "ggml_mul_mat_vec_a8");
}
Tensor ggml_mul_mat_a8(const Tensor& W, const Tensor& X, int64_t type, int64_t row) {
  return matmul_common(W, X, type, row, GGUF_B200_OP_MMQ, "ggml_mul_mat_a8");
}
Tensor dequant_matmul(const Tensor& W, const Tensor& X, int64_t type, int64_t row) {
  return matmul_common(W, X, type, row, GGUF_B200_OP_DEQUANT_MATMUL, "dequant_matmul");
}

Tensor ggml_moe_a8(const Tensor& X, const Tensor& W, const Tensor& sorted_token_ids, const Tensor& expert_ids,
                   const Tensor& num_tokens_post_padded, int64_t type, int64_t row, int64_t top_k, int64_t tokens) {
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t K = check_weight(W, type, "ggml_moe_a8");
  TORCH_CHECK(W.dim() == 3, "ggml_moe_a8: W must be [experts, rows, bytes]");
  TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == K, "ggml_moe_a8: X must be contiguous [tokens, K]");
  TORCH_CHECK(X.size(0) == tokens, "ggml_moe_a8: X.shape[0] != tokens");
  TORCH_CHECK(row == W.size(1), "ggml_moe_a8: row != W.shape[1]");
  TORCH_CHECK(sorted_token_ids.scalar_type() == ScalarType::Int && expert_ids.scalar_type() == ScalarType::Int &&
                  num_tokens_post_padded.scalar_type() == ScalarType::Int,
              "ggml_moe_a8: routing tensors must be int32");
  TORCH_CHECK(sorted_token_ids.is_contiguous() && expert_ids.is_contiguous(), "ggml_moe_a8: routing tensors must be contiguous");
  const int blk = gguf_b200_moe_block_size((int)type);
  TORCH_CHECK(blk > 0, "ggml_moe_a8: type has no tensor-core MoE kernel");
  const int64_t n_sorted = sorted_token_ids.numel();
  // vLLM sizes sorted_token_ids as numel + E*(block-1) (not rounded) and expert_ids as its ceil-div by block
  TORCH_CHECK(expert_ids.numel() * blk >= n_sorted,
              "ggml_moe_a8: sorted_token_ids/expert_ids were not built with block size ggml_moe_get_block_size(type)");
  const int code = dtype_code(X.scalar_type(), "ggml_moe_a8");
  Tensor Y = new_tensor({tokens * top_k, row}, X.scalar_type(), X.device());  // zeroed by the C-ABI call
  const int64_t ws_bytes = gguf_b200_scratch_bytes(GGUF_B200_OP_MOE, (int)type, n_sorted, row, K);
  const Scratch ws(ws_bytes);
  check_rc(gguf_b200_moe_a8(X.data_ptr(), W.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes,
                            static_cast<const int32_t*>(sorted_token_ids.data_ptr()), static_cast<const int32_t*>(expert_ids.data_ptr()),
                            static_cast<const int32_t*>(num_tokens_post_padded.data_ptr()), n_sorted, W.stride(0),
                            W.size(0) < 256 ? W.size(0) : 256,   // ids beyond 255 are skipped, as in the reference (moe.cuh:33)
                            (int)type, code, tokens, top_k, row, K, current_stream(X.get_device())),
           "ggml_moe_a8");
  return Y;
}

Tensor ggml_moe_a8_vec(const Tensor& X, const Tensor& W, const Tensor& topk_ids, int64_t top_k, int64_t type, int64_t row, int64_t tokens) {
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t K = check_weight(W, type, "ggml_moe_a8_vec");
  TORCH_CHECK(W.dim() == 3 && row == W.size(1), "ggml_moe_a8_vec: W must be [experts, row, bytes]");
  TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == K && X.size(0) == tokens, "ggml_moe_a8_vec: X must be contiguous [tokens, K]");
  TORCH_CHECK(topk_ids.scalar_type() == ScalarType::Int && topk_ids.is_contiguous() && topk_ids.numel() == tokens * top_k,
              "ggml_moe_a8_vec: topk_ids must be contiguous int32 [tokens, top_k]");
  const int code = dtype_code(X.scalar_type(), "ggml_moe_a8_vec");
  Tensor Y = new_tensor({tokens * top_k, row}, X.scalar_type(), X.device());
  if (tokens == 0 || row == 0) return Y;
  const int64_t ws_bytes = gguf_b200_workspace_bytes(GGUF_B200_OP_MOE_VEC, (int)type, tokens, row, K);
  const Scratch ws(ws_bytes);
  check_rc(gguf_b200_moe_a8_vec(X.data_ptr(), W.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, static_cast<const int32_t*>(topk_ids.data_ptr()),
                                W.size(0), (int)type, code, tokens, top_k, row, K, current_stream(X.get_device())),
           "ggml_moe_a8_vec");
  return Y;
}

// The MoE step in one call (see gguf_b200_fused_moe).  act: 1 silu, 2 gelu.
Tensor fused_moe(const Tensor& X, const Tensor& W13, const Tensor& W2, const Tensor& topk_weights, const Tensor& topk_ids, int64_t type13,
                 int64_t type2, int64_t act) {
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t H = check_weight(W13, type13, "fused_moe");
  const int64_t I = check_weight(W2, type2, "fused_moe");
  TORCH_CHECK(W13.dim() == 3 && W2.dim() == 3 && W13.size(0) == W2.size(0), "fused_moe: W13 / W2 must be [experts, rows, bytes]");
  TORCH_CHECK(W13.size(1) == 2 * I && W2.size(1) == H, "fused_moe: W13 must be [E, 2I, .] and W2 [E, H, .]");
  TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == H, "fused_moe: X must be contiguous [tokens, H]");
  TORCH_CHECK(topk_ids.scalar_type() == ScalarType::Int && topk_ids.is_contiguous() && topk_ids.dim() == 2 && topk_ids.size(0) == X.size(0),
              "fused_moe: topk_ids must be contiguous int32 [tokens, top_k]");
  TORCH_CHECK(topk_weights.scalar_type() == ScalarType::Float && topk_weights.is_contiguous() && topk_weights.numel() == topk_ids.numel(),
              "fused_moe: topk_weights must be contiguous float32 [tokens, top_k]");
  const int code = dtype_code(X.scalar_type(), "fused_moe");
  const int64_t tokens = X.size(0), top_k = topk_ids.size(1), E = W13.size(0);
  Tensor Y = new_tensor({tokens, H}, X.scalar_type(), X.device());
  const int64_t ws_bytes = gguf_b200_fused_moe_workspace_bytes((int)type13, (int)type2, code, tokens, top_k, E, H, I);
  TORCH_CHECK(ws_bytes > 0 || tokens == 0, "fused_moe: unsupported types or sizes");
  const Scratch ws(ws_bytes);
  check_rc(gguf_b200_fused_moe(X.data_ptr(), W13.data_ptr(), W2.data_ptr(), Y.data_ptr(), static_cast<const int32_t*>(topk_ids.data_ptr()),
                               static_cast<const float*>(topk_weights.data_ptr()), ws.get(), ws_bytes, (int)type13, (int)type2, code, (int)act,
                               tokens, top_k, E, H, I, current_stream(X.get_device())),
           "fused_moe");
  return Y;
}

int64_t ggml_moe_get_block_size(int64_t type) { return gguf_b200_moe_block_size((int)type); }

TORCH_LIBRARY(_C_gguf, ops) {
  ops.def("ggml_dequantize(Tensor W, int type, SymInt m, SymInt n, ScalarType? dtype) -> Tensor");
  ops.def("ggml_mul_mat_vec_a8(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def("ggml_mul_mat_a8(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def(
      "ggml_moe_a8(Tensor X, Tensor W, Tensor sorted_token_ids, Tensor expert_ids, Tensor num_tokens_post_padded, "
      "int type, SymInt row, SymInt top_k, SymInt tokens) -> Tensor");
  ops.def("ggml_moe_a8_vec(Tensor X, Tensor W, Tensor topk_ids, int top_k, int type, SymInt row, SymInt tokens) -> Tensor");
  ops.def("ggml_moe_get_block_size(int type) -> int");
  ops.def("dequant_matmul(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def("dequantize_rows(Tensor W, Tensor ids, int type, ScalarType? dtype) -> Tensor");
  ops.def("fused_moe(Tensor X, Tensor W13, Tensor W2, Tensor topk_weights, Tensor topk_ids, int type13, int type2, int act) -> Tensor");
}

TORCH_LIBRARY_IMPL(_C_gguf, CUDA, ops) {
  ops.impl("ggml_dequantize", &ggml_dequantize);
  ops.impl("ggml_mul_mat_vec_a8", &ggml_mul_mat_vec_a8);
  ops.impl("ggml_mul_mat_a8", &ggml_mul_mat_a8);
  ops.impl("ggml_moe_a8", &ggml_moe_a8);
  ops.impl("ggml_moe_a8_vec", &ggml_moe_a8_vec);
  ops.impl("dequant_matmul", &dequant_matmul);
  ops.impl("dequantize_rows", &dequantize_rows);
  ops.impl("fused_moe", &fused_moe);
}

TORCH_LIBRARY_IMPL(_C_gguf, CompositeExplicitAutograd, ops) { ops.impl("ggml_moe_get_block_size", &ggml_moe_get_block_size); }

// ---- eager calls ---------------------------------------------------------------------------------

namespace {

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
  return THPVariable_Wrap(matmul_common(*W, *X, type, row, (int)op, names[op]));
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
  const c10::cuda::CUDAGuard guard(W->device());
  const int64_t K = check_weight(*W, type, "embed");
  if (K != hidden || K % 256 != 0 || ids->device() != W->device()) Py_RETURN_NONE;
  const int code = dtype_code(dt, "embed");
  c10::SmallVector<int64_t, 4> shape(ids->sizes().begin(), ids->sizes().end());
  shape.push_back(hidden);
  Tensor out = new_tensor(shape, dt, W->device());
  rows_into(*W, *ids, type, K, out, code);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// The batch-size rule of the linear dispatcher (quantization/linear.py `_fused_mul_mat_gguf`): the
// operation that serves M rows against N weight rows of `type`, or -1 where only Python does.
bool imatrix_type(int64_t t) { return t == 16 || t == 17 || t == 18 || t == 19 || t == 20 || t == 21 || t == 22 || t == 23 || t == 29; }
int linear_op(int64_t type, int64_t M, int64_t N, ScalarType dt) {
  const bool im = imatrix_type(type);
  const int64_t most = im ? (N > 5120 ? 8 : 16) : (N > 5120 ? 2 : 6);
  if (M <= most) return GGUF_B200_OP_GEMV;
  if (!im) return GGUF_B200_OP_MMQ;
  const bool fused = dt == ScalarType::Half || dt == ScalarType::BFloat16;
  return fused ? GGUF_B200_OP_DEQUANT_MATMUL : -1;
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
  const int op = linear_op(type, X->size(0), N, X->scalar_type());
  if (op < 0) Py_RETURN_NONE;
  return THPVariable_Wrap(matmul_common(*W, *X, type, N, op, "linear"));
  END_HANDLE_TH_ERRORS
}

// linear_runs(x, W, runs): a layer whose rows are of several types, stacked in W and padded to its width.  runs: a flat tuple of
// (type, first row, rows, bytes of a row, rows that decide the routing) per run.  Every run is multiplied where it lies, into its columns of one result.
PyObject* py_linear_runs(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 3 && PyTuple_Check(a[2]) && PyTuple_GET_SIZE(a[2]) % 5 == 0, "linear_runs takes x, W and a tuple of runs");
  const Tensor *X = plain_cuda(a[0]), *W = plain_cuda(a[1]);
  if (!W || !X || X->dim() != 2 || W->dim() != 2 || X->size(0) == 0 || !modes_off() || !X->is_contiguous() || !W->is_contiguous() ||
      W->scalar_type() != ScalarType::Byte)
    Py_RETURN_NONE;
  const ScalarType dt = X->scalar_type();
  if (dt != ScalarType::Float && dt != ScalarType::Half && dt != ScalarType::BFloat16) Py_RETURN_NONE;
  struct Run { int type, op; int64_t row, rows, ws; };
  c10::SmallVector<Run, 4> runs;
  const int64_t M = X->size(0), K = X->size(1), pitch = W->size(1);
  int64_t N = 0, most = 0;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[2]); i += 5) {
    long v[5];
    for (int j = 0; j < 5; ++j) v[j] = PyLong_AsLong(PyTuple_GET_ITEM(a[2], i + j));
    if (PyErr_Occurred()) return nullptr;
    const int ts = gguf_b200_type_size((int)v[0]);
    if (ts == 0 || v[3] % ts != 0 || v[3] / ts * gguf_b200_block_size((int)v[0]) != K || v[1] < 0 || v[1] + v[2] > W->size(0) || v[1] * pitch % 16 != 0)
      Py_RETURN_NONE;
    const int op = linear_op(v[0], M, v[4], dt);
    if (op < 0) Py_RETURN_NONE;
    const int64_t ws = gguf_b200_scratch_bytes(op, (int)v[0], M, v[2], K);
    most = ws > most ? ws : most;
    runs.push_back({(int)v[0], op, v[1], v[2], ws});
    N += v[2];
  }
  if (N == 0) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(X->device());
  Tensor Y = new_tensor({M, N}, dt, X->device());
  const Scratch ws(most);
  const int code = dtype_code(dt, "linear_runs");
  void* s = current_stream(X->get_device());
  int64_t col = 0;
  for (const Run& r : runs) {
    uint8_t* y = static_cast<uint8_t*>(Y.data_ptr()) + col * Y.element_size();
    if (reinterpret_cast<uintptr_t>(y) % 16 != 0) Py_RETURN_NONE;
    const int rc = gguf_b200_mul_mat_strided(static_cast<const uint8_t*>(W->data_ptr()) + r.row * pitch, X->data_ptr(), y, ws.get(), most, r.op, r.type,
                                             code, M, r.rows, K, pitch, N, s);
    if (rc == GGUF_B200_E_SHAPE || rc == GGUF_B200_E_TOO_LARGE) Py_RETURN_NONE;   // a layout that only copies can serve
    check_rc(rc, "linear_runs");
    col += r.rows;
  }
  return THPVariable_Wrap(std::move(Y));
  END_HANDLE_TH_ERRORS
}

// moe(x, W13, W2, topk_weights, topk_ids, type13, type2, act): the whole expert step
PyObject* py_moe(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "moe takes 8 arguments");
  const Tensor* t[5];
  for (int i = 0; i < 5; ++i)
    if (!(t[i] = plain_cuda(a[i]))) Py_RETURN_NONE;
  if (!modes_off()) Py_RETURN_NONE;
  const long type13 = PyLong_AsLong(a[5]), type2 = PyLong_AsLong(a[6]), act = PyLong_AsLong(a[7]);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(fused_moe(*t[0], *t[1], *t[2], *t[3], *t[4], type13, type2, act));
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
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_C_gguf", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyObject* PyInit__C_gguf(void) { return PyModule_Create(&module_def); }
