// Internal launcher declarations shared by the translation units of libgguf_b200.
// (The public C-ABI is include/gguf_b200.h; nothing here is exported.)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gguf_b200 {

// output layouts of the q8_1 quantizer (quantize_q8_1.cu)
enum : int { Q8_MODE_REF = 0, Q8_MODE_SOA = 1, Q8_MODE_F16 = 2 };
// correction column appended to the fp16 activation matrix of the tensor-core kernels
enum : int { CORR_NONE = 0, CORR_Q4_0 = 1, CORR_MIN = 2, CORR_PLUS = 3 };   // B-side column: 8*(d8*sum(q8) - s8), -s8, +s8

// Tensor-parallel input of the SoA quantizer (one vector).  A gathered vector lives on every rank
// as "packets": one 32-bit word {16-bit value, 16-bit tag} per element for f16/bf16 outputs, one
// 64-bit word {f32 value, 32-bit tag} for f32, each written by a single store of the producing
// GEMV (possibly on another GPU).  The quantizer reads x'[k] = x[k] + add_scale * value(add[k])
// (x may be null), polling every packet until its tag equals *add_epoch (bounded by limit_cycles,
// then *status = E_TIMEOUT).  bump != null: thread 0 of the grid increments *bump first -- the
// launch number of the GEMV that follows, which that GEMV uses as the tag of its own packets.
struct Q8Tp {
  const void* add = nullptr;        // packets of the vector to add (element type = the x dtype), or null
  const unsigned* add_epoch = nullptr;
  float add_scale = 0.f;
  int add_parts = 1;                // > 1: the slot holds that many fp32 partial vectors (a row-parallel call's), add_stride
  int64_t add_stride = 0;           //      packets apart; their sum, taken in rank order, is the vector that is added
  unsigned* bump = nullptr;
  int early = 0;                    // the product behind the quantizer may read its weights before work ahead of both is complete
  long long limit_cycles = 0;
  int* status = nullptr;
};
// M = number of OUTPUT rows.  gather_ids (F16 mode only, may be null): output row r quantizes
// input row gather_ids[r] / gather_div; ids outside [0, gather_limit) give a zero row.
int launch_quantize_q8_1(const void* x, int x_dtype, void* out, int64_t M, int64_t K, int mode, int sum_mode,
                         int64_t ldb, int corr_mode, const int32_t* gather_ids, int64_t gather_div, int64_t gather_limit,
                         cudaStream_t stream, int perm = 0, const Q8Tp* tp = nullptr, int act = 0, int64_t x_ld = 0,
                         int* zero = nullptr, int64_t n_zero = 0, const int32_t* n_used = nullptr);
// zero, n_zero (F16 mode, aligned rows): words to clear for the kernel behind it; n_used: [1] = rows of the output in use (null: M).
// act (F16 mode): 0 = none; 1 = silu, 2 = gelu: the input rows are [gate | up] of x_ld = 2K values and act(gate) * up is quantized
// leading dimension (elements) of the fp16 activation matrix of the tensor-core kernels
int64_t mmq_ldb(int type, int64_t K);
int mmq_corr_mode(int type);
// value order the tensor-core kernel will expect in the fp16 activation matrix for this problem
int mmq_perm(int type, int64_t K, int64_t pitch, bool gap);   // gap: between one expert's matrix and the next

// row_ids != null: row gather -- out row r (K values, K a multiple of 256) = weight row row_ids[r] of weight_rows
int launch_dequantize(const void* w, int type, void* out, int out_dtype, int64_t n_elems, int q4k_contract,
                      cudaStream_t stream, const int64_t* row_ids = nullptr, int64_t K = 0, int64_t weight_rows = 0);

// Fused dequant-GEMV over SoA q8_1 activations (see quantize_q8_1.cu for the layout).
// Y[m, n] for m in [0, M); rows of W are N x (K/QK*TS) bytes, contiguous, 16-byte aligned base.
int launch_gemv(const void* w, const void* xq_soa, void* y, int type, int out_dtype, int64_t M, int64_t N, int64_t K,
                int* status, cudaStream_t stream);
// The whole decode op for M <= 2 vectors in ONE launch (activations quantized inside the GEMV kernel);
// returns 1 when the shape needs the two-kernel route.
int launch_gemv_fused(const void* w, const void* x, void* y, int type, int dtype, int64_t M, int64_t N, int64_t K, int sum_mode,
                      int* status, cudaStream_t stream, int64_t pitch = 0, bool w_in_flight = false);
// One- and two-vector specialisation (gemv1.cu): activations in registers.  Returns 1 when the
// shape is outside its reach (the caller then uses the general kernel).
// Tensor-parallel output of the single-vector kernel: every result is sent to all `world` ranks
// as a packet at ll_peer[r] + y_off + row (see Q8Tp), tagged with epoch[slot].
struct GemvTp {
  int world, slot;
  const unsigned* epoch;    // this rank's launch counters (incremented by the quantizer before the launch)
  int64_t y_off;
  void* ll_peer[8];
};
// MoE decode through the same kernel: y row s = weights of expert topk_ids[s] (N x K each, back
// to back) times activation vector s / top_k of the `tokens` quantized ones
struct GemvMoe {
  const int32_t* topk_ids;
  int64_t tokens, top_k, n_experts, slots;
};
int launch_gemv1(const void* w, const void* xq_soa, void* y, int type, int out_dtype, int64_t N, int64_t K, int* status,
                 cudaStream_t stream, const GemvTp* tp = nullptr, int vectors = 1, const GemvMoe* moe = nullptr,
                 int vec0 = 0, int total_vecs = 0,    // vec0 / total_vecs: the `vectors` handled are vec0.. of total_vecs in the scratch
                 const void* x_raw = nullptr, int x_sum_mode = 0, int64_t pitch = 0, int64_t ldy = 0,    // 0: rows back to back, ldy = N
                 bool w_in_flight = false);   // the work ahead may still write w: no byte of it is read before that is complete
// x_raw != null (element type = out_dtype): the activations [vectors or tokens][K] are NOT quantized yet and xq_soa is
// ignored -- every CTA quantizes what it needs in shared memory (one launch per GEMV); returns 1 if that does not fit.
// 1 when the q8_1 scratch of this type's GEMV must hold d * sum(q) instead of the fp16 sum of the inputs
inline int gemv_sum_mode(int type) { return (type == 12 || type == 13) ? 1 : 0; }   // Q4_K, Q5_K
// Packets of `nslots` gathered vectors (slot_packets apart) -> plain vectors out[s][0..n) (out_stride
// elements apart); every packet is polled until its tag equals epoch[slot0 + s] (bounded).
// one thread waits (bounded) until flag[slot] has reached world * epoch[slot]
int launch_tp_wait(const unsigned* flag, const unsigned* epoch, int slot, int world, long long limit_cycles, int* status,
                   cudaStream_t stream);
int launch_tp_unpack(const void* packets, const unsigned* epoch, int slot0, int nslots, int64_t slot_packets, int64_t n,
                     void* out, int64_t out_stride, int dtype, long long limit_cycles, int* status, cudaStream_t stream);
int launch_tp_unpack_sum(const void* packets, const unsigned* epoch, int slot, int64_t slot_bytes, int64_t n, int parts, void* out,
                         int dtype, long long limit_cycles, int* status, cudaStream_t stream);
// per-(token,expert) GEMV of the small-batch MoE entry point
int launch_moe_gemv(const void* w, const void* xq_soa, void* y, const int32_t* topk_ids, int type, int out_dtype,
                    int64_t tokens, int64_t top_k, int64_t N, int64_t K, int64_t n_experts, int* status,
                    cudaStream_t stream);

// Tensor-core (tcgen05) dequant-GEMM.  B operand = fp16/bf16 matrix [rows][ldb] (K-major).
// Tensor-parallel output of the tensor-core GEMM: this rank's [M][N] result is column block
// [col_off, col_off + N) of a gathered [M][ld] matrix that every rank holds; the kernel stores its
// tiles into ALL ranks' copies (y_peer[r], plain 16-byte stores over NVLink, this rank included),
// and the last CTA to finish increments epoch[slot] and then flag_peer[r][slot] on every rank.
struct MmqTp {
  int world, slot;
  int64_t col_off, ld;
  unsigned* epoch;
  void* y_peer[8];
  unsigned* flag_peer[8];
};
struct MmqArgs {
  const void* w;            // packed weights (expert 0), rows `pitch` bytes apart
  const void* b;            // activation matrix, K-major, element type b_dtype (DT_F16 / DT_BF16), ldb elements between rows
  void* y;                  // output, element type out_dtype, ldy elements between rows
  int type, out_dtype, b_dtype;
  int64_t M;                // activation rows
  int64_t N, K;             // weight rows, values per row
  int64_t pitch, ldb, ldy;
  int corr_mode;            // which correction the columns behind K hold
  int perm;                 // value order of b (see mmq_perm)
  // MoE (null passes = dense): the work list of launch_moe_plan / launch_moe_blocks
  const void* passes;       // int4 {expert, first activation row, rows}
  const int32_t* n_passes;
  const int32_t* sorted;    // output row of every activation row (>= rows_out: padding)
  int64_t experts, max_passes, pass_rows, rows_out;
  int64_t expert_gap;       // MoE: bytes between one expert's matrix and the next
  const float* row_scale;   // MoE: output row r is multiplied by row_scale[r] (routing weights); null: no scaling
  int* status;
  const MmqTp* tp;          // null: plain output y
  bool w_in_flight;         // no quantizer is ahead and earlier work may still write w (see pdl_wait)
  // Optional: room for tiles that several CTAs share (mmq_share).  `counter` must be zero when the kernel starts.
  int* counter;
  int64_t zero_counters;    // > 0: so many words of it are cleared here first
  void* part;               // 16-byte aligned, part_bytes long
  int64_t part_bytes;
};
int launch_mmq(const MmqArgs& a, cudaStream_t stream);
// scratch with which every CTA gets an equal share of the chunks: n_counters words, then partial tiles
struct MmqShare { int64_t n_counters, counter_bytes, part_bytes; };
MmqShare mmq_share(int type, int64_t M, int64_t N, int64_t K);   // all zero where sharing does not pay
MmqShare mmq_share_moe(int64_t N, int64_t max_passes, int64_t pass_rows);
int launch_zero(int* p, int64_t n, cudaStream_t stream);
int launch_fence(cudaStream_t stream);   // an empty kernel in plain stream order (see pdl_wait)
int mmq_moe_block_size();

int64_t q8_soa_bytes(int64_t M, int64_t K);

// Small-batch product on the 8-bit tensor instruction (smallm.cu), dense or per expert.  The activations are quantized into
// tiles of eight columns by launch_quantize_frag, which launch_smallm calls first.
struct SmallArgs {
  const void* w;             // packed weights (expert 0), rows `pitch` bytes apart
  const void* x;             // activations, element type dtype
  void* y;                   // element type dtype, rows ldy elements apart
  void* ws;                  // smallm_scratch_bytes(tiles, max_passes, n, k), 256-byte aligned
  int type, dtype, sum_mode; // sum_mode: see gemv_sum_mode
  int64_t m, n, k;           // tokens (dense), weight rows, values per row
  int64_t pitch, ldy;
  int64_t tiles;             // column tiles of eight (MoE: room for)
  int64_t experts, max_passes;   // dense: 1, 1
  // MoE (null passes = dense): written on the device by launch_moe_plan
  const void* passes;        // int4 {expert, first column tile, column tiles, 0}
  const int32_t* n_passes;   // [0] passes, [1] column tiles in use
  const int32_t* sorted;     // output row of every column, rows_out in padding columns
  int pass_tiles;            // column tiles of a pass (1, 2 or 4)
  int64_t rows_out;
  int64_t x_div;             // column c takes activation row sorted[c] / x_div
  int act;                   // 1 silu, 2 gelu: the rows of x are [gate | up] of 2k values (see launch_quantize_q8_1)
  const float* row_scale;
  int* status;
};
int launch_smallm(const SmallArgs& a, cudaStream_t stream);
int launch_quantize_frag(const SmallArgs& a, void* out, int* counters, int64_t n_counters, cudaStream_t stream);
int64_t smallm_scratch_bytes(int64_t tiles, int64_t passes, int64_t n, int64_t k);
int smallm_max_tokens();
int smallm_table_bytes(int type);
bool smallm_pairs_with_sum(int type);
int smallm_order(int type);      // order of a block's values in the tiles (smallm_decode.cuh)

// fused MoE step (moe_fused.cu)
// The routed slots (token * top_k + j) sorted by expert, every expert's run starting at a multiple of `align` rows, and a work list
// of passes of up to pass_rows rows of one expert.  passes: int4 {expert, first row / align, rows / align rounded up (align > 1) or
// rows, 0}; sorted[row] = slot, `slots` in padding rows; n_passes: [0] passes, [1] rows in use / align.
int64_t moe_plan_rows(int64_t slots, int n_experts, int align);              // room for rows
int64_t moe_plan_passes(int64_t slots, int n_experts, int pass_rows);
int launch_moe_plan(const int32_t* topk_ids, int64_t slots, int n_experts, int align, int pass_rows, int32_t* sorted, void* passes,
                    int32_t* n_passes, cudaStream_t stream);
// passes of `block` rows from a caller's block-aligned lists (expert ids outside [0, n_experts) and blocks beyond n_post_pad left out)
int launch_moe_blocks(const int32_t* expert_ids, const int32_t* n_post_pad, int64_t n_sorted, int n_experts, int block, void* passes,
                      int32_t* n_passes, cudaStream_t stream);
int launch_moe_sum(const void* y, void* out, const int32_t* topk_ids, int n_experts, int64_t tokens, int64_t top_k, int64_t h,
                   int dtype, cudaStream_t stream);

// Device address of the library's one status word on the current device (the word that
// gguf_b200_last_status reads and clears); null if the runtime refuses the lookup.
int* status_word_ptr();

}  // namespace gguf_b200
