// Small-batch product  Y[m, n] = sum_k dequant(W)[n, k] * q8_1(X)[m, k]  for batches of a few tokens, dense and per expert:
// the decode GEMV entry points from three tokens on (reference: mul_mat_vec_q, mmvq.cuh:2-41; moe_vec_q, moe_vec.cuh) and
// ggml_mul_mat_a8 for the batches that are bound by reading the weights.
//
// Arithmetic: the integer dot products of the reference's vec_dot_*_q8_1, on the 8-bit tensor instruction
// mma.sync.m16n8k32 (16 weight rows x 32 values against eight tokens; exact), then the format's scales in fp32 on the CUDA
// cores.  At these batches the instruction count decides, not the tensor rate: one instruction replaces the 128 dp4a of a
// 16 x 32 block and eight tokens, a block's codes are unpacked once for all tokens, and what is left per block, token
// tile and lane is 8 (no minimum) to 12 floating-point instructions.  (tcgen05 needs the codes as a 128-row operand in
// tensor memory and the scales folded into 16-bit operands; its instruction costs at least 25 clocks however few tokens it
// has, and the fp16 rounding of the operands is not what this entry point promises.)
//
// Work: a CTA (eight warps x 16 rows, one warp that issues copies) streams stages of 256 values x 128 rows (raw_stream.cuh)
// together with the activation tiles of the same 256 values.  The units (row tile, chunk) of the whole matrix are dealt out
// as equal contiguous ranges, whatever the shape: a row tile that several CTAs share is added up by the last of them to
// arrive, in chunk order (deterministic; the partial tiles stay in L2).  Two CTAs per SM.
//
// Measured (B200, device time per call, activations included; before: the dp4a kernels, two or eight tokens per pass): Q4_K 14336x4096, 4 / 8 /
// 16 tokens 20.7 / 37.3 / 76.0 -> 16.3 / 16.0 / 20.1 us; Q6_K 28.7 / 55.0 / 111 -> 21.8 / 21.7 / 28.2; IQ4_XS 30.0 / 43.2 / 89.7 -> 21.0 / 20.5 / 24.3.
#include "smallm.cuh"

namespace gguf_b200 {

#define SM_EXTERN(TYPE) extern template int sm_launch<TYPE>(const SmParams&, const CUtensorMap&, int, int, size_t, cudaStream_t);
#define SM_TYPES(X) X(T_Q4_0) X(T_Q4_1) X(T_Q5_0) X(T_Q5_1) X(T_Q8_0) X(T_Q2_K) X(T_Q3_K) X(T_Q4_K) X(T_Q5_K) X(T_Q6_K) X(T_IQ2_XXS) X(T_IQ2_XS) \
  X(T_IQ2_S) X(T_IQ3_XXS) X(T_IQ3_S) X(T_IQ1_S) X(T_IQ1_M) X(T_IQ4_NL) X(T_IQ4_XS)
SM_TYPES(SM_EXTERN)

// Column tiles per CTA pass; the kernel is compiled for 1, 2 and 4.
static int sm_t(int tiles) { return tiles <= 1 ? 1 : tiles <= 2 ? 2 : 4; }
int smallm_max_tokens() { return 32; }

constexpr int SM_GRID = 2 * 148;
static int64_t sm_x_bytes(int64_t tiles, int64_t K) { return (K + RAW_KC - 1) / RAW_KC * tiles * SM_TILE_BYTES; }
static int64_t sm_part_bytes(int t) { return (int64_t)2 * SM_GRID * SM_WARPS * 32 * t * 16; }
static int64_t sm_counter_bytes(int64_t passes, int64_t N) { return round_up(passes * ((N + RAW_ROWS - 1) / RAW_ROWS) * 4, 256); }

int64_t smallm_scratch_bytes(int64_t tiles, int64_t passes, int64_t N, int64_t K) {
  return round_up(sm_x_bytes(tiles, K), 256) + sm_counter_bytes(passes, N) + sm_part_bytes(sm_t((int)(tiles < 4 ? tiles : 4)));
}

int launch_smallm(const SmallArgs& a, cudaStream_t stream) {
  if (a.n == 0 || a.tiles == 0) return E_OK;
  SmParams p{};
  CUtensorMap map{};
  if (!plan_raw(a.type, a.w, a.n, a.experts, a.k, a.pitch, p.raw, map)) return E_BAD_SHAPE;
  const int t = a.passes ? a.pass_tiles : sm_t(a.tiles);
  uint8_t* ws = static_cast<uint8_t*>(a.ws);
  p.w = static_cast<const uint8_t*>(a.w);
  p.w_bytes = (a.n * a.experts - 1) * a.pitch + p.raw.row_bytes;
  p.x = ws;
  p.counter = reinterpret_cast<int*>(ws + round_up(sm_x_bytes(a.tiles, a.k), 256));
  p.part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.counter) + sm_counter_bytes(a.max_passes, a.n));
  p.y = a.y;
  p.ldy = a.ldy;
  p.dtype = a.dtype;
  p.n = (int)a.n;
  p.m = (int)a.m;
  p.nblk = (int)(a.k / 32);
  p.nc = (int)((a.k + RAW_KC - 1) / RAW_KC);
  p.rt = (int)((a.n + RAW_ROWS - 1) / RAW_ROWS);
  p.tiles = (int)a.tiles;
  p.status = a.status;
  p.passes = static_cast<const int4*>(a.passes);
  p.n_passes = a.n_passes;
  p.sorted = a.sorted;
  p.rows_out = (int)a.rows_out;
  p.row_scale = a.row_scale;
  // activations -> 8-bit tiles (and the arrival counters to zero)
  int rc = launch_quantize_frag(a, ws, p.counter, sm_counter_bytes(a.max_passes, a.n) / 4, stream);
  if (rc) return rc;
  p.stage_bytes = p.raw.bytes + (int)((a.passes ? t : a.tiles) * SM_TILE_BYTES);
  const int table = smallm_table_bytes(a.type);
  int stages = (int)((113 * 1024 - 256 - table) / p.stage_bytes);   // two CTAs per SM
  if (stages > SM_MAX_STAGES) stages = SM_MAX_STAGES;
  if (stages < 2) return E_TOO_LARGE;
  p.stages = stages;
  // A CTA asks for up to 60 KB of weights at a time.  The memory system serves what is outstanding interleaved: with whole rings asked
  // for -- most of a 33 MB matrix -- every CTA's first stage arrived with the last, 3.6 us into the wait (14336x4096, eight tokens, all / four /
  // three / two / one stage: Q4_K, 18 KB a stage, 17.4 / 16.7 / 16.2 / 15.7 / 16.4 us; Q6_K, 31 KB, 22.9 / 22.7 / 22.8 / 21.8 / 21.1).
  p.ahead = 60 * 1024 / p.raw.bytes;
  p.ahead = p.ahead < 1 ? 1 : p.ahead > stages ? stages : p.ahead;
  const size_t smem = 256 + (size_t)table + (size_t)stages * p.stage_bytes;
  const int64_t units = (int64_t)a.max_passes * p.rt * p.nc;
  if (units * (SM_GRID + 1) >= (int64_t)1 << 31) return E_TOO_LARGE;
  const int grid = (int)(units < SM_GRID ? units : SM_GRID);
  switch (a.type) {
#define SM_CASE(TYPE) case TYPE: return sm_launch<TYPE>(p, map, t, grid, smem, stream);
    SM_TYPES(SM_CASE)
  }
  return E_BAD_TYPE;
}

int smallm_table_bytes(int type) {
  switch (type) {
#define SM_TAB(TYPE) case TYPE: return sm_table_bytes<TYPE>();
    SM_TYPES(SM_TAB)
  }
  return 0;
}
bool smallm_pairs_with_sum(int type) { return sm_pairs_with_sum(type); }
int smallm_order(int type) { return sm_order(type); }

}  // namespace gguf_b200
