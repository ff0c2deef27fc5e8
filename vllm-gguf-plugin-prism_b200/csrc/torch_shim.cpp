// Torch library `_C_gguf` over the C-ABI of libgguf_b200: the six operator schemas of the
// reference's binding file (vllm_gguf_plugin/csrc/torch_bindings.cpp:22-53), registered the same
// way (stable ABI, ops on the CUDA key, ggml_moe_get_block_size as CompositeExplicitAutograd), so
// `vllm_gguf_plugin.ops` finds `torch.ops._C_gguf.*` unchanged, plus dequant_matmul (the fused route
// of the IQ types), dequantize_rows, fused_moe and linear_runs.  The bodies are in op_calls.h.
//
// This file uses nothing of torch but its stable ABI and nothing of Python but the module
// entry: the library runs under every torch that has that ABI, whatever the Python version.
// (The functions that eager calls go through need more than that: eager.cpp, a module of its own.)
#include <Python.h>
#include <torch/csrc/inductor/aoti_torch/c/shim.h>
#include <torch/csrc/stable/accelerator.h>
#include <torch/csrc/stable/library.h>
#include <torch/csrc/stable/ops.h>
#include <torch/csrc/stable/tensor.h>

#include <vector>

#include "op_calls.h"

namespace {

struct Stable {
  using Tensor = torch::stable::Tensor;
  using Guard = torch::stable::accelerator::DeviceGuard;
  static int32_t device(const Tensor& t) { return t.get_device_index(); }
  static void* stream(const Tensor& t) {
    void* raw = nullptr;
    TORCH_ERROR_CODE_CHECK(aoti_torch_get_current_cuda_stream(device(t), &raw));
    return raw;
  }
  static Tensor empty(const Tensor& like, std::initializer_list<int64_t> sizes, torch::headeronly::ScalarType t) {
    return torch::stable::new_empty(like, sizes, t);
  }
  static bool has_room(const Tensor& t, int64_t bytes) {
    int64_t size = 0, offset = 0;
    TORCH_ERROR_CODE_CHECK(aoti_torch_get_storage_size(t.get(), &size));
    TORCH_ERROR_CODE_CHECK(aoti_torch_get_storage_offset(t.get(), &offset));
    return size - offset >= bytes;
  }
  static Tensor block(Tensor t, int64_t row, int64_t rows, int64_t col, int64_t cols) {
    Tensor r = torch::stable::narrow(t, 0, row, rows);
    return torch::stable::narrow(r, 1, col, cols);
  }
  static Tensor packed(const Tensor& t) { return torch::stable::contiguous(t); }
  static void copy(Tensor to, const Tensor& from) { torch::stable::copy_(to, from); }
  struct Scratch {
    Tensor t;
    Scratch(const Tensor& like, int64_t bytes) : t(empty(like, {bytes > 0 ? bytes : 1}, torch::headeronly::ScalarType::Byte)) {}
    void* get() const { return t.data_ptr(); }
  };
};
using Tensor = Stable::Tensor;
using Op = gguf_ops::Calls<Stable>;
using torch::headeronly::ScalarType;

Tensor ggml_dequantize(Tensor W, int64_t type, int64_t m, int64_t n, std::optional<ScalarType> dtype) { return Op::dequantize(W, type, m, n, dtype); }
Tensor dequantize_rows(Tensor W, Tensor ids, int64_t type, std::optional<ScalarType> dtype) { return Op::dequantize_rows(W, ids, type, dtype); }
Tensor ggml_mul_mat_vec_a8(Tensor W, Tensor X, int64_t type, int64_t row) { return Op::mul_mat(W, X, type, row, GGUF_B200_OP_GEMV, "ggml_mul_mat_vec_a8", false); }
Tensor ggml_mul_mat_a8(Tensor W, Tensor X, int64_t type, int64_t row) { return Op::mul_mat(W, X, type, row, GGUF_B200_OP_MMQ, "ggml_mul_mat_a8", false); }
Tensor dequant_matmul(Tensor W, Tensor X, int64_t type, int64_t row) { return Op::mul_mat(W, X, type, row, GGUF_B200_OP_DEQUANT_MATMUL, "dequant_matmul", false); }
Tensor ggml_moe_a8(Tensor X, Tensor W, Tensor sorted_token_ids, Tensor expert_ids, Tensor num_tokens_post_padded, int64_t type, int64_t row,
                   int64_t top_k, int64_t tokens) {
  return Op::moe_a8(X, W, sorted_token_ids, expert_ids, num_tokens_post_padded, type, row, top_k, tokens);
}
Tensor ggml_moe_a8_vec(Tensor X, Tensor W, Tensor topk_ids, int64_t top_k, int64_t type, int64_t row, int64_t tokens) {
  return Op::moe_a8_vec(X, W, topk_ids, top_k, type, row, tokens);
}
Tensor fused_moe(Tensor X, Tensor W13, Tensor W2, Tensor topk_weights, Tensor topk_ids, int64_t type13, int64_t type2, int64_t act) {
  return Op::fused_moe(X, W13, W2, topk_weights, topk_ids, type13, type2, act);
}
Tensor linear_runs(Tensor X, Tensor W, std::vector<int64_t> runs) { return Op::linear_runs(X, W, runs.data(), runs.size()); }
void weights_complete(Tensor W) { Op::weights_complete(W); }
int64_t ggml_moe_get_block_size(int64_t type) { return gguf_b200_moe_block_size((int)type); }

}  // namespace

STABLE_TORCH_LIBRARY(_C_gguf, ops) {
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
  ops.def("weights_complete(Tensor W) -> ()");
  ops.def("linear_runs(Tensor X, Tensor W, int[] runs) -> Tensor");
  ops.def("fused_moe(Tensor X, Tensor W13, Tensor W2, Tensor topk_weights, Tensor topk_ids, int type13, int type2, int act) -> Tensor");
}

STABLE_TORCH_LIBRARY_IMPL(_C_gguf, CUDA, ops) {
  ops.impl("ggml_dequantize", TORCH_BOX(&ggml_dequantize));
  ops.impl("ggml_mul_mat_vec_a8", TORCH_BOX(&ggml_mul_mat_vec_a8));
  ops.impl("ggml_mul_mat_a8", TORCH_BOX(&ggml_mul_mat_a8));
  ops.impl("ggml_moe_a8", TORCH_BOX(&ggml_moe_a8));
  ops.impl("ggml_moe_a8_vec", TORCH_BOX(&ggml_moe_a8_vec));
  ops.impl("dequant_matmul", TORCH_BOX(&dequant_matmul));
  ops.impl("dequantize_rows", TORCH_BOX(&dequantize_rows));
  ops.impl("weights_complete", TORCH_BOX(&weights_complete));
  ops.impl("linear_runs", TORCH_BOX(&linear_runs));
  ops.impl("fused_moe", TORCH_BOX(&fused_moe));
}

STABLE_TORCH_LIBRARY_IMPL(_C_gguf, CompositeExplicitAutograd, ops) { ops.impl("ggml_moe_get_block_size", TORCH_BOX(&ggml_moe_get_block_size)); }

static PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_C_gguf", nullptr, -1, nullptr};
extern "C" PyObject* PyInit__C_gguf(void) { return PyModule_Create(&module_def); }
