// What an operator does between its tensors and the C-ABI (gguf_b200.h): validates the tensors, allocates the output and
// the scratch memory from torch's caching allocator (so CUDA-graph capture works as in the reference), resolves the
// current stream and turns error codes into exceptions.  All arithmetic lives behind gguf_b200.h.
//
// Written once for the two tensor types it is called with (A): torch's stable ABI (torch_shim.cpp, the registered
// operators) and at::Tensor (eager.cpp, the functions of an eager call).  A gives the tensor type, a device guard, `empty`,
// `device`, `stream` and a `Scratch` that holds the memory of one call.
#pragma once

#include <optional>
#include <string>

#include <torch/headeronly/core/ScalarType.h>
#include <torch/headeronly/util/Exception.h>

#include "../../include/gguf_b200.h"

namespace gguf_ops {

using torch::headeronly::ScalarType;

inline int dtype_code(ScalarType t, const char* what) {
  switch (t) {
    case ScalarType::Float: return GGUF_B200_F32;
    case ScalarType::Half: return GGUF_B200_F16;
    case ScalarType::BFloat16: return GGUF_B200_BF16;
    default: break;
  }
  STD_TORCH_CHECK(false, what, ": expected a float32, float16 or bfloat16 tensor");
  return -1;
}

inline void check_rc(int rc, const char* op) { STD_TORCH_CHECK(rc == GGUF_B200_OK, op, " failed: ", gguf_b200_error_string(rc)); }

// The batch-size rule of the linear dispatcher (quantization/linear.py `_fused_mul_mat_gguf`): the
// operation that serves M rows against N weight rows of `type`, or -1 where only Python does.
inline bool imatrix_type(int64_t t) { return t == 16 || t == 17 || t == 18 || t == 19 || t == 20 || t == 21 || t == 22 || t == 23 || t == 29; }
inline int linear_op(int64_t type, int64_t M, int64_t N, ScalarType dt) {
  const bool im = imatrix_type(type);
  const int64_t most = im ? (N > 5120 ? 8 : 16) : (N > 5120 ? 2 : 6);
  if (M <= most) return GGUF_B200_OP_GEMV;
  if (!im) return GGUF_B200_OP_MMQ;
  const bool fused = dt == ScalarType::Half || dt == ScalarType::BFloat16;
  return fused ? GGUF_B200_OP_DEQUANT_MATMUL : -1;
}

template <class A> struct Calls {
  using Tensor = typename A::Tensor;

  // Weights are raw GGUF bytes: uint8, contiguous, last dim a whole number of blocks.
  static int64_t check_weight(const Tensor& W, int64_t type, const char* op) {
    const int ts = gguf_b200_type_size((int)type);
    STD_TORCH_CHECK(ts > 0, op, ": unsupported GGML quantization type ", std::to_string(type));
    STD_TORCH_CHECK(W.scalar_type() == ScalarType::Byte, op, ": W must be a uint8 tensor of raw GGUF blocks");
    STD_TORCH_CHECK(W.is_contiguous(), op, ": W must be contiguous");
    STD_TORCH_CHECK(W.dim() >= 1 && W.size(W.dim() - 1) % ts == 0, op, ": last dim of W is not a whole number of blocks");
    return W.size(W.dim() - 1) / ts * gguf_b200_block_size((int)type);  // K
  }

  static Tensor dequantize(const Tensor& W, int64_t type, int64_t m, int64_t n, std::optional<ScalarType> dtype) {
    const typename A::Guard guard(A::device(W));
    check_weight(W, type, "ggml_dequantize");
    const ScalarType dt = dtype.value_or(ScalarType::Half);
    const int code = dtype_code(dt, "ggml_dequantize");
    const int ts = gguf_b200_type_size((int)type), bs = gguf_b200_block_size((int)type);
    STD_TORCH_CHECK(m >= 0 && n >= 0 && (m * n) % bs == 0, "ggml_dequantize: m*n must be a multiple of the block size");
    STD_TORCH_CHECK(W.numel() >= m * n / bs * ts, "ggml_dequantize: W holds fewer than m*n values");
    Tensor out = A::empty(W, {m, n}, dt);  // every element is written by the kernel
    check_rc(gguf_b200_dequantize(W.data_ptr(), (int)type, out.data_ptr(), code, m * n, A::stream(W)), "ggml_dequantize");
    return out;
  }

  // rows `ids` (contiguous int64, any shape) of the packed weight into `out`
  static void rows_into(const Tensor& W, const Tensor& ids, int64_t type, int64_t K, const Tensor& out, int code) {
    check_rc(gguf_b200_dequantize_rows(W.data_ptr(), (int)type, static_cast<const int64_t*>(ids.data_ptr()), ids.numel(), K, W.size(0),
                                       out.data_ptr(), code, A::stream(W)),
             "dequantize_rows");
  }

  // Embedding look-up: rows `ids` of the packed weight, dequantized (replaces index_select +
  // ggml_dequantize of the reference's embedding caller, quantization/vocal_embeds.py:88-96).
  static Tensor dequantize_rows(const Tensor& W, const Tensor& ids, int64_t type, std::optional<ScalarType> dtype) {
    const typename A::Guard guard(A::device(W));
    const int64_t K = check_weight(W, type, "dequantize_rows");
    STD_TORCH_CHECK(W.dim() == 2, "dequantize_rows: W must be [rows, bytes]");
    STD_TORCH_CHECK(ids.scalar_type() == ScalarType::Long && ids.is_contiguous() && ids.dim() == 1,
                    "dequantize_rows: ids must be a contiguous 1-D int64 tensor");
    STD_TORCH_CHECK(K % 256 == 0, "dequantize_rows: the row length must be a multiple of 256");
    const ScalarType dt = dtype.value_or(ScalarType::Half);
    const int code = dtype_code(dt, "dequantize_rows");
    Tensor out = A::empty(W, {ids.size(0), K}, dt);
    rows_into(W, ids, type, K, out, code);
    return out;
  }

  // The three dense products (op: GGUF_B200_OP_GEMV, _MMQ, _DEQUANT_MATMUL).  settled: W is a loaded layer's weight, complete
  // since its loading; any other tensor may come straight out of a kernel, and the calls that read weights ahead of the
  // stream are told so.
  static Tensor mul_mat(const Tensor& W, const Tensor& X, int64_t type, int64_t row, int op, const char* name, bool settled) {
    const typename A::Guard guard(A::device(X));
    const int64_t K = check_weight(W, type, name);
    STD_TORCH_CHECK(X.dim() == 2 && X.is_contiguous(), name, ": X must be a contiguous [tokens, K] tensor");
    STD_TORCH_CHECK(X.size(1) == K, name, ": X.shape[1] does not match the K implied by W");
    STD_TORCH_CHECK(row >= 0 && W.numel() / W.size(W.dim() - 1) >= row, name, ": W has fewer than `row` rows");
    const int code = dtype_code(X.scalar_type(), name);
    const int64_t M = X.size(0);
    Tensor Y = A::empty(X, {M, row}, X.scalar_type());
    if (M == 0 || row == 0) return Y;
    const int64_t ws_bytes = gguf_b200_scratch_bytes(op, (int)type, M, row, K);
    const typename A::Scratch ws(X, ws_bytes);
    void* s = A::stream(X);
    int rc = GGUF_B200_E_TOO_LARGE;
    if (!settled && (op == GGUF_B200_OP_DEQUANT_MATMUL || (op == GGUF_B200_OP_GEMV && M <= 2)))
      rc = gguf_b200_mul_mat_strided(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, op | GGUF_B200_W_IN_FLIGHT, (int)type, code, M, row,
                                     K, W.size(W.dim() - 1), row, s);
    if (rc != GGUF_B200_E_TOO_LARGE)
      ;
    else if (!settled && op == GGUF_B200_OP_GEMV && M <= 2)   // rows too long for that form
      check_rc(gguf_b200_weights_complete(s), name), rc = gguf_b200_mul_mat_vec_a8(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
    else if (op == GGUF_B200_OP_GEMV)
      rc = gguf_b200_mul_mat_vec_a8(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
    else if (op == GGUF_B200_OP_MMQ)
      rc = gguf_b200_mul_mat_a8(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
    else
      rc = gguf_b200_dequant_matmul(W.data_ptr(), X.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, (int)type, code, M, row, K, s);
    check_rc(rc, name);
    return Y;
  }

  // A loaded layer's product.  Its rows may be of several types, stacked in W [rows, bytes of the widest] a stride apart; runs: (type,
  // first row, rows, bytes of a row, rows that decide the routing) of each run of one type.  Every run is multiplied where it lies, into
  // its columns of one result.  What the kernels cannot do in place -- columns off a 16-byte boundary, a row distance that the
  // format cannot be read at, rows too long for them -- is multiplied into, or as, a copy.
  static Tensor linear_runs(const Tensor& X, const Tensor& W, const int64_t* runs, size_t n) {
    const char* name = "linear_runs";
    const typename A::Guard guard(A::device(X));
    STD_TORCH_CHECK(n > 0 && n % 5 == 0, name, ": five numbers per run");
    STD_TORCH_CHECK(W.scalar_type() == ScalarType::Byte && W.dim() == 2 && W.stride(1) == 1, name, ": W must be uint8 rows of raw GGUF blocks");
    STD_TORCH_CHECK(X.dim() == 2 && X.is_contiguous(), name, ": X must be a contiguous [tokens, K] tensor");
    const ScalarType dt = X.scalar_type();
    const int code = dtype_code(dt, name);
    const int64_t M = X.size(0), K = X.size(1), pitch = W.stride(0), esz = dt == ScalarType::Float ? 4 : 2;
    int64_t N = 0, ws_bytes = 0;
    for (size_t i = 0; i < n; i += 5) {
      const int64_t *r = runs + i, ts = gguf_b200_type_size((int)r[0]);
      STD_TORCH_CHECK(ts > 0, name, ": unsupported GGML quantization type ", std::to_string(r[0]));
      STD_TORCH_CHECK(r[1] >= 0 && r[2] >= 0 && r[1] + r[2] <= W.size(0) && r[3] <= W.size(1) && r[3] % ts == 0 && r[3] / ts * gguf_b200_block_size((int)r[0]) == K,
                      name, ": a run does not match X and W");
      const int op = linear_op(r[0], M, r[4], dt);
      STD_TORCH_CHECK(op >= 0, name, ": no kernel for this type, batch and dtype");
      const int64_t ws = M > 0 ? gguf_b200_scratch_bytes(op, (int)r[0], M, r[2], K) : 0;
      ws_bytes = ws > ws_bytes ? ws : ws_bytes;
      N += r[2];
    }
    Tensor Y = A::empty(X, {M, N}, dt);
    if (M == 0 || N == 0) return Y;
    const typename A::Scratch ws(X, ws_bytes);
    void* s = A::stream(X);
    // (every row is followed by the bytes up to the next, the last one, too)
    const bool in_place = pitch >= W.size(1) && A::has_room(W, W.size(0) * pitch);
    int64_t col = 0;
    for (size_t i = 0; i < n; i += 5) {
      const int64_t *r = runs + i, rows = r[2];
      if (rows == 0) continue;
      const int type = (int)r[0], op = linear_op(r[0], M, r[4], dt);
      uint8_t* y = static_cast<uint8_t*>(Y.data_ptr()) + col * esz;
      const uint8_t* w = static_cast<const uint8_t*>(W.data_ptr()) + r[1] * pitch;
      const bool direct = reinterpret_cast<uintptr_t>(y) % 16 == 0;
      std::optional<Tensor> part;
      if (!direct) part = A::empty(X, {M, rows}, dt);
      int rc = GGUF_B200_E_SHAPE;
      if (in_place && reinterpret_cast<uintptr_t>(w) % 16 == 0)
        rc = gguf_b200_mul_mat_strided(w, X.data_ptr(), direct ? y : part->data_ptr(), ws.get(), ws_bytes, op, type, code, M, rows, K, pitch,
                                       direct ? N : rows, s);
      if (rc == GGUF_B200_E_SHAPE || rc == GGUF_B200_E_TOO_LARGE) {
        part = mul_mat(A::packed(A::block(W, r[1], rows, 0, r[3])), X, type, rows, op, name, false);
        rc = GGUF_B200_OK;
      }
      check_rc(rc, name);
      if (part) A::copy(A::block(Y, 0, M, col, rows), *part);
      col += rows;
    }
    return Y;
  }

  static void weights_complete(const Tensor& W) {
    const typename A::Guard guard(A::device(W));
    check_rc(gguf_b200_weights_complete(A::stream(W)), "weights_complete");
  }

  static Tensor moe_a8(const Tensor& X, const Tensor& W, const Tensor& sorted_token_ids, const Tensor& expert_ids,
                       const Tensor& num_tokens_post_padded, int64_t type, int64_t row, int64_t top_k, int64_t tokens) {
    const typename A::Guard guard(A::device(X));
    const int64_t K = check_weight(W, type, "ggml_moe_a8");
    STD_TORCH_CHECK(W.dim() == 3, "ggml_moe_a8: W must be [experts, rows, bytes]");
    STD_TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == K, "ggml_moe_a8: X must be contiguous [tokens, K]");
    STD_TORCH_CHECK(X.size(0) == tokens, "ggml_moe_a8: X.shape[0] != tokens");
    STD_TORCH_CHECK(row == W.size(1), "ggml_moe_a8: row != W.shape[1]");
    STD_TORCH_CHECK(sorted_token_ids.scalar_type() == ScalarType::Int && expert_ids.scalar_type() == ScalarType::Int &&
                        num_tokens_post_padded.scalar_type() == ScalarType::Int,
                    "ggml_moe_a8: routing tensors must be int32");
    STD_TORCH_CHECK(sorted_token_ids.is_contiguous() && expert_ids.is_contiguous(), "ggml_moe_a8: routing tensors must be contiguous");
    const int blk = gguf_b200_moe_block_size((int)type);
    STD_TORCH_CHECK(blk > 0, "ggml_moe_a8: type has no tensor-core MoE kernel");
    const int64_t n_sorted = sorted_token_ids.numel();
    // vLLM sizes sorted_token_ids as numel + E*(block-1) (not rounded) and expert_ids as its ceil-div by block
    STD_TORCH_CHECK(expert_ids.numel() * blk >= n_sorted,
                    "ggml_moe_a8: sorted_token_ids/expert_ids were not built with block size ggml_moe_get_block_size(type)");
    const int code = dtype_code(X.scalar_type(), "ggml_moe_a8");
    Tensor Y = A::empty(X, {tokens * top_k, row}, X.scalar_type());  // zeroed by the C-ABI call
    const int64_t ws_bytes = gguf_b200_scratch_bytes(GGUF_B200_OP_MOE, (int)type, n_sorted, row, K);
    const typename A::Scratch ws(X, ws_bytes);
    check_rc(gguf_b200_moe_a8(X.data_ptr(), W.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes,
                              static_cast<const int32_t*>(sorted_token_ids.data_ptr()), static_cast<const int32_t*>(expert_ids.data_ptr()),
                              static_cast<const int32_t*>(num_tokens_post_padded.data_ptr()), n_sorted, W.stride(0),
                              W.size(0) < 256 ? W.size(0) : 256,   // ids beyond 255 are skipped, as in the reference (moe.cuh:33)
                              (int)type, code, tokens, top_k, row, K, A::stream(X)),
             "ggml_moe_a8");
    return Y;
  }

  static Tensor moe_a8_vec(const Tensor& X, const Tensor& W, const Tensor& topk_ids, int64_t top_k, int64_t type, int64_t row, int64_t tokens) {
    const typename A::Guard guard(A::device(X));
    const int64_t K = check_weight(W, type, "ggml_moe_a8_vec");
    STD_TORCH_CHECK(W.dim() == 3 && row == W.size(1), "ggml_moe_a8_vec: W must be [experts, row, bytes]");
    STD_TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == K && X.size(0) == tokens, "ggml_moe_a8_vec: X must be contiguous [tokens, K]");
    STD_TORCH_CHECK(topk_ids.scalar_type() == ScalarType::Int && topk_ids.is_contiguous() && topk_ids.numel() == tokens * top_k,
                    "ggml_moe_a8_vec: topk_ids must be contiguous int32 [tokens, top_k]");
    const int code = dtype_code(X.scalar_type(), "ggml_moe_a8_vec");
    Tensor Y = A::empty(X, {tokens * top_k, row}, X.scalar_type());
    if (tokens == 0 || row == 0) return Y;
    const int64_t ws_bytes = gguf_b200_workspace_bytes(GGUF_B200_OP_MOE_VEC, (int)type, tokens, row, K);
    const typename A::Scratch ws(X, ws_bytes);
    check_rc(gguf_b200_moe_a8_vec(X.data_ptr(), W.data_ptr(), Y.data_ptr(), ws.get(), ws_bytes, static_cast<const int32_t*>(topk_ids.data_ptr()),
                                  W.size(0), (int)type, code, tokens, top_k, row, K, A::stream(X)),
             "ggml_moe_a8_vec");
    return Y;
  }

  // The MoE step in one call (see gguf_b200_fused_moe).  act: 1 silu, 2 gelu.
  static Tensor fused_moe(const Tensor& X, const Tensor& W13, const Tensor& W2, const Tensor& topk_weights, const Tensor& topk_ids, int64_t type13,
                          int64_t type2, int64_t act) {
    const typename A::Guard guard(A::device(X));
    const int64_t H = check_weight(W13, type13, "fused_moe");
    const int64_t I = check_weight(W2, type2, "fused_moe");
    STD_TORCH_CHECK(W13.dim() == 3 && W2.dim() == 3 && W13.size(0) == W2.size(0), "fused_moe: W13 / W2 must be [experts, rows, bytes]");
    STD_TORCH_CHECK(W13.size(1) == 2 * I && W2.size(1) == H, "fused_moe: W13 must be [E, 2I, .] and W2 [E, H, .]");
    STD_TORCH_CHECK(X.dim() == 2 && X.is_contiguous() && X.size(1) == H, "fused_moe: X must be contiguous [tokens, H]");
    STD_TORCH_CHECK(topk_ids.scalar_type() == ScalarType::Int && topk_ids.is_contiguous() && topk_ids.dim() == 2 && topk_ids.size(0) == X.size(0),
                    "fused_moe: topk_ids must be contiguous int32 [tokens, top_k]");
    STD_TORCH_CHECK(topk_weights.scalar_type() == ScalarType::Float && topk_weights.is_contiguous() && topk_weights.numel() == topk_ids.numel(),
                    "fused_moe: topk_weights must be contiguous float32 [tokens, top_k]");
    const int code = dtype_code(X.scalar_type(), "fused_moe");
    const int64_t tokens = X.size(0), top_k = topk_ids.size(1), E = W13.size(0);
    Tensor Y = A::empty(X, {tokens, H}, X.scalar_type());
    const int64_t ws_bytes = gguf_b200_fused_moe_workspace_bytes((int)type13, (int)type2, code, tokens, top_k, E, H, I);
    STD_TORCH_CHECK(ws_bytes > 0 || tokens == 0, "fused_moe: unsupported types or sizes");
    const typename A::Scratch ws(X, ws_bytes);
    check_rc(gguf_b200_fused_moe(X.data_ptr(), W13.data_ptr(), W2.data_ptr(), Y.data_ptr(), static_cast<const int32_t*>(topk_ids.data_ptr()),
                                 static_cast<const float*>(topk_weights.data_ptr()), ws.get(), ws_bytes, (int)type13, (int)type2, code, (int)act,
                                 tokens, top_k, E, H, I, A::stream(X)),
             "fused_moe");
    return Y;
  }
};

}  // namespace gguf_ops
