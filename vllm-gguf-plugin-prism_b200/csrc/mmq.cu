// Prefill GEMM on the 5th-generation tensor cores:  D[n, t] = sum_k A[n, k] * B[t, k]
// with A = weight tile decoded on the fly from packed GGUF blocks and B = activations.
// Serves three entry points:
//   * ggml_mul_mat_a8   (reference: gguf_kernel.cu:220-290 + mul_mat_q, mmq.cuh:2-104)
//   * ggml_moe_a8       (reference: gguf_kernel.cu:292-393 + moe_q, moe.cuh:5-129)
//   * dequantize-then-matmul of the IQ types (reference: quantization/linear.py:50-54)
//
// Why fp16 operands and not int8: the contraction carries a different fp scale per 32
// values on BOTH operands (weights: d or d*sc; activations: the q8_1 d).  An int8 MMA would
// have to drain its int32 accumulator and rescale it on the CUDA cores after every K=32 step
// (128 x 256 accumulators per ~130 tensor clocks), which bounds it near 10-25 % of int8 peak.
// Folding the scales into the operands instead -- A = half(scale * code) decoded exactly as
// the reference's own dequantize does, B = half(d8 * q8) from the bit-exact q8_1 quantizer --
// keeps ONE fp32 accumulator in tensor memory over the whole K with no drain, at the price of
// one fp16 rounding per operand (~3e-4 relative L2, far inside the 2e-3 budget).  The q8_1
// "sum" terms the reference's tiled kernels use (Q4_0: -8*d*s8, Q4_K: -dmin*m*s8, with s8 the
// fp16 sum of the *unquantized* activations) ride along as K/32 extra contraction columns.
//
// Tile: 128 weight rows (UMMA M) x tn tokens (any multiple of 16 up to 256, two instructions side by side up to 384) x 64 values
// per stage.  Operand A (the decoded weights) lives in tensor memory: a producer thread owns one weight row = one lane, and
// stores the 64 fp16 values of a stage -- 32 registers -- into 32 columns of that lane with tcgen05.st; the MMA takes A from
// there ([a_tmem] operand form).  Operand B (activations) is K-major in shared memory with the 128-byte swizzle, one TMA box per
// stage.  Weight rows sit on the M axis so that small token counts do not waste the 128-row instruction.
//
// Warp roles: 16 producer warps in four groups of 128 threads, which take items -- half chunks, two stages -- in turn and also read
// the accumulators out; a B loader, an MMA issuer, a raw-weight loader.  An item has one full/empty barrier pair; up to 128
// tokens a tile its activations arrive on it too, in one box.  Every wait is bounded in time and reports through the status word.
// The correction values are taken from the raw chunk while it is decoded and written to shared memory as a tile of operand A; the
// tensor core multiplies it once per four chunks (gathered from global memory at the end of a tile they took 10,600 clocks of it).
//
// One CTA per SM lives for the whole launch, over a range of (tile, 256-value chunk) units (mmq_plan); a tile that several CTAs
// share is added up by the last of them to arrive, in CTA order (deterministic).  While a tile's accumulator is read out the
// loaders, the decoders (an item per group) and, with two accumulators, the tensor core are already at work on the next one.
//
// What bounded the kernel before (one CTA per tile, 64 stages of a tile; clocks taken inside it, Q4_K 14336 x 4096): 5,700
// clocks passed before a tile's first MMA and 4,800 in its epilogue, of 46,700 at 512 tokens; at 32 tokens a stage took 445
// clocks because a B slot came back 745 clocks after its MMA and refilling it took 1,050 more, over a ring of four.
// tcgen05.mma itself takes max(25, tn / 2) clocks per 16 values when its operands are in uniform registers, 119 to 147 from a loop that the
// compiler takes for divergent; a wait that is ready, with its address arithmetic, 80 to 250.  With an MMA issuer of the second sort
// and three waits an item, no type got below 460 to 560 clocks a stage; since its warp stays converged and waits once, the decoders
// bound the kernel at 128 tokens or less.  Clocks a stage at 48 tokens, before -> after: Q4_K 511 -> 326, Q4_0 490 -> 313, Q2_K 562 -> 397,
// Q5_K 542 -> 429, IQ2_XXS 621 -> 459, Q3_K 684 -> 465, Q6_K 717 -> 405 (its unit decoder 537).
// Measured, before -> after: IQ3_S 8192 x 28672, 300 tokens 291 -> 134 us; Q6_K 37888 x 3584, 1999 tokens 668 -> 567 us;
// IQ2_XXS 28672 x 8192, 128 tokens 108 -> 95 us; a MoE step of 256 tokens (64 experts, Q4_0) 222 -> 169 us.  By items and with the
// converged issuer: Q6_K 3584 x 18944, 45 tokens 36.5 -> 28.0 us; the MoE step 167.6 -> 142.3; IQ2_XXS 92.5 -> 79.1; Q6_K 1999 tokens 546 -> 503.
#include "mmq_kernel.cuh"

namespace gguf_b200 {

#define MMQ_TYPES(X) X(T_Q4_0) X(T_Q4_1) X(T_Q5_0) X(T_Q5_1) X(T_Q8_0) X(T_Q2_K) X(T_Q3_K) X(T_Q4_K) X(T_Q5_K) X(T_Q6_K) X(T_IQ2_XXS) X(T_IQ2_XS) \
  X(T_IQ2_S) X(T_IQ3_XXS) X(T_IQ3_S) X(T_IQ1_S) X(T_IQ1_M) X(T_IQ4_NL) X(T_IQ4_XS)
#define MMQ_EXTERN(TYPE) \
  extern template int mmq_launch<TYPE>(const MmqParams&, const CUtensorMap&, const CUtensorMap&, int, bool, int, size_t, cudaStream_t);
MMQ_TYPES(MMQ_EXTERN)

constexpr int MMQ_CTAS = 148;

int mmq_moe_block_size() { return 64; }

// The whole-stage decoders read dense stages, and want the activations in the order of their nibbles.  One decision, shared
// by the activation quantizer and the launch.
static bool mmq_fast(int type, int64_t K, int64_t pitch) {
  return (type == T_Q4_0 || type == T_Q8_0 || type == T_Q4_K || type == T_Q5_K) && raw_dense(type, K, pitch);
}
// The order of the values in the activation matrix: 0 as they are; 1, inside every four 0, 2, 1, 3; 2, inside every four blocks of 32
// the blocks 0, 2, 1, 3 (Item128<T_Q6_K>).
int mmq_perm(int type, int64_t K, int64_t pitch, bool gap) {
  if (type == T_Q6_K) return 2;
  return !gap && mmq_fast(type, K, pitch) && type != T_Q8_0 ? 1 : 0;
}
static_assert(Stage64<T_Q4_0, __half>::PERM == 1 && Stage64<T_Q4_K, __half>::PERM == 1 && Stage64<T_Q5_K, __half>::PERM == 1 &&
                  Stage64<T_Q8_0, __half>::PERM == 0,
              "mmq_perm");

// How a dense problem is dealt out, by the clocks it should take.  The tokens are split over `tt` tiles of `tn`; the tiles go
// to the CTAs, one per SM, in one of three ways:
//   whole    every tile is one CTA's
//   even     few tiles: each is cut into the same number of ranges of chunks, one per CTA
//   stream   the chunks of all tiles in equal runs over all SMs
// A stage takes the time to decode it (mmq_decode_clocks) or that of its product and its activations (mmq_stage_clocks); reading a tile
// out takes 13.5 clocks per token, 6 where there are two accumulators (beside the next tile's work); a CTA in use 50; sharing, 1,800 + 44 per
// token + 11 per token and part where a CTA has one part of a tile, 7,000 + 34 per token + 16.5 per token and part where it has two (6,300 by
// the times of graphs of one product; between other work 512 tokens of 14336x4096 Q4_K take 67.4 us in whole tiles and 68.3 in runs).
// Fitted by least squares, then by what is lost, to the times of every plan of 3,500 problems (19 types, eight matrices of 1024x4096 to
// 28672x8192, 17 to 1999 tokens, weights from memory, plans timed in turn; those beyond 256 tokens on three GPUs, which the power limit holds back
// to different degrees): what it picks takes 0.5 % longer than the best plan on average, 15 % at most.  (The clocks before these had tiles of
// more than 256 tokens too long by a tenth and those of up to 256 too short: 300 tokens of 8192x28672 Q8_0 were cut into two tiles, 157 us
// where one takes 137; 700 of 37888x3584 IQ2_S into three, 151 where two take 145.)
struct MmqPlan {
  int tn;
  int64_t tt, grid;
  bool shared;
};
// clocks to decode a stage, with what a CTA of many tokens leaves of its issue slots and shared memory (half a clock per token).  One number a type,
// between those of fp16 and bf16 activations (IQ4_XS 560 and 620, IQ4_NL 570 and 650, alike or within 1 % for the others): a workspace's size
// follows from the plan, and the caller who asks for it names no activation type.
static int mmq_decode_clocks(int type) {
  switch (type) {
    case T_Q8_0: return 300;
    case T_Q4_K: return 305;
    case T_Q4_0: return 310;
    case T_Q4_1: return 425;
    case T_Q2_K: return 430;
    case T_IQ2_XXS: return 445;
    case T_Q6_K: return 450;
    case T_IQ2_S: return 460;
    case T_Q5_0: case T_Q5_1: case T_Q5_K: case T_IQ2_XS: return 475;
    case T_IQ1_S: return 480;
    case T_IQ3_XXS: case T_IQ3_S: return 490;
    case T_Q3_K: return 510;
    case T_IQ1_M: return 530;
    case T_IQ4_XS: return 590;
    default: return 610;   // IQ4_NL
  }
}
// (the product itself takes two clocks per token; the rest is the activations' way from L2 and, beyond 256 tokens, the few A slots)
static int64_t mmq_stage_clocks(int type, int tn) {
  const int decode = mmq_decode_clocks(type) + (tn <= 256 ? tn : 256) / 2;
  const int mma = tn <= 128 ? 250 + 3 * tn / 2 : tn <= 256 ? 190 + 7 * tn / 4 : tn <= 320 ? 300 + 13 * tn / 8 : 170 + 33 * tn / 16;
  return mma > decode ? mma : decode;
}
static MmqPlan mmq_plan(int type, int64_t M, int64_t N, int64_t K, bool may_share) {
  const int64_t rt = (N + MMQ_ROWS - 1) / MMQ_ROWS, nc = (K + RAW_KC - 1) / RAW_KC;
  MmqPlan best{};
  int64_t best_t = INT64_MAX, last = 0;
  // tiles as large as the tensor memory allows, or of one instruction, or with two accumulators -- and somewhat smaller ones
  const struct { int64_t cap, more; } sizes[3] = {{384, 4}, {256, 3}, {128, 3}};
  for (const auto& z : sizes) {
    for (int64_t tt = (int64_t)((uint32_t)(M + z.cap - 1) / (uint32_t)z.cap), e = tt + z.more; tt < e; ++tt) {
      if (tt <= last || tt > M) continue;
      last = tt;
      const int64_t rows = (uint32_t)(M + tt - 1) / (uint32_t)tt;
      const int tn = (int)round_up(rows, rows > 256 ? 32 : 16);
      if ((uint32_t)(M + tn - 1) / (uint32_t)tn < tt) continue;   // (rounded up, fewer tiles do)
      const int64_t tiles = rt * tt, chunk = 4 * mmq_stage_clocks(type, tn), waves = (tiles + MMQ_CTAS - 1) / MMQ_CTAS;
      const bool twin = tn <= 128;
      auto take = [&](int64_t t, int64_t grid, bool shared) {
        t += 50 * grid;
        if (t < best_t) { best_t = t; best = {tn, tt, grid, shared}; }
      };
      take(waves * nc * chunk + (twin ? 12 : waves * 27) * tn / 2, tiles < MMQ_CTAS ? tiles : MMQ_CTAS, false);
      if (!may_share) continue;
      if (tiles % MMQ_CTAS != 0 && tiles * nc >= 2 * MMQ_CTAS) {
        const int64_t run = (tiles * nc + MMQ_CTAS - 1) / MMQ_CTAS;
        take(run * chunk + (twin ? 12 : (tiles / MMQ_CTAS + 1) * 27) * tn / 2 + 7000 + 34 * tn + 33 * tn * nc / (2 * run), MMQ_CTAS, true);
      }
      // (32-bit divisions: a call asks for its plan three times; a cut into more ranges of the same length only costs)
      const int ncs = (int)nc;
      for (int c = 2, len = 0; c * tiles <= MMQ_CTAS && 2 * c <= ncs; ++c) {
        const int l = (ncs + c - 1) / c;
        if (l != len) take((int64_t)l * chunk + 1800 + tn * (44 + 11 * c), c * tiles, true);
        len = l;
      }
    }
  }
  return best;
}

MmqShare mmq_share(int type, int64_t M, int64_t N, int64_t K) {
  MmqShare s{};
  if (M <= 0 || N <= 0 || K <= 0) return s;
  const MmqPlan pl = mmq_plan(type, M, N, K, true);
  if (!pl.shared) return s;
  s.n_counters = (N + MMQ_ROWS - 1) / MMQ_ROWS * pl.tt;
  s.counter_bytes = round_up(s.n_counters * 4, 256);
  s.part_bytes = 2 * pl.grid * MMQ_ROWS * pl.tn * 4;
  return s;
}
MmqShare mmq_share_moe(int64_t N, int64_t max_passes, int64_t pass_rows) {
  MmqShare s{};
  s.n_counters = (N + MMQ_ROWS - 1) / MMQ_ROWS * max_passes;
  s.counter_bytes = round_up(s.n_counters * 4, 256);
  s.part_bytes = (int64_t)2 * MMQ_CTAS * MMQ_ROWS * round_up(pass_rows, 16) * 4;
  return s;
}

__global__ void __launch_bounds__(256) zero_kernel(int* p, int64_t n) {
  pdl_trigger();
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = 0;
}
int launch_zero(int* p, int64_t n, cudaStream_t stream) {
  if (n <= 0) return E_OK;
  return launch_pdl(zero_kernel, dim3((unsigned)((n + 255) / 256 > 64 ? 64 : (n + 255) / 256)), dim3(256), 0, stream, p, n) == cudaSuccess ? E_OK : E_CUDA;
}

__global__ void fence_kernel() {}
int launch_fence(cudaStream_t stream) {
  fence_kernel<<<1, 1, 0, stream>>>();
  return cudaGetLastError() == cudaSuccess ? E_OK : E_CUDA;
}

// Three activation boxes of the largest tile have to fit beside the tables and two raw stages of rows of any pitch (an odd number of
// 16-byte units each, with the rows that a class map leaves over).  With two, 1152 tokens of 37888x3584 IQ3_XXS took 281 us instead of 231.
template <int TYPE> constexpr bool mmq_three_boxes() {
  constexpr int units = (RAW_KC / BlockTraits<TYPE>::QK * BlockTraits<TYPE>::TS + 30) / 16 | 1;
  constexpr int raw = (RAW_ROWS + RAW_EXTRA) * units * 16 + 128, corr = Decoder<TYPE, __half>::CORR ? MMQ_CORR_BYTES : 0;
  return 226 * 1024 - 512 - decoder_table_bytes<TYPE>() - corr - 2 * raw >= 3 * 384 * MMQ_BK * 2;
}
#define MMQ_FITS(TYPE) static_assert(mmq_three_boxes<TYPE>(), #TYPE);
MMQ_TYPES(MMQ_FITS)

static int mmq_aux_bytes(int type) {   // barriers, then the decoder's tables
  switch (type) {
#define MMQ_TAB(TYPE) case TYPE: return 512 + decoder_table_bytes<TYPE>();
    MMQ_TYPES(MMQ_TAB)
  }
  return 512;
}
int launch_mmq(const MmqArgs& a, cudaStream_t stream) {
  if (a.N == 0 || a.M == 0) return E_OK;
  const bool bf = a.b_dtype == DT_BF16;
  MmqParams p{};
  CUtensorMap wmap{}, bmap{};
  if (!plan_raw(a.type, a.w, a.N, a.passes ? a.experts : 1, a.K, a.pitch, p.raw, wmap, a.expert_gap)) return E_BAD_SHAPE;
  const bool fast = mmq_fast(a.type, a.K, a.pitch) && p.raw.mode == 1;
  if (a.perm != mmq_perm(a.type, a.K, a.pitch, !fast)) return E_BAD_SHAPE;
  p.w = static_cast<const uint8_t*>(a.w);
  p.w_bytes = (a.N * (a.passes ? a.experts : 1) - 1) * a.pitch + p.raw.row_bytes + (a.passes ? (a.experts - 1) * p.raw.gap : 0);
  p.y = a.y;
  p.ldy = a.ldy;
  p.dtype = a.out_dtype;
  p.n = (int)a.N;
  p.m = (int)a.M;
  p.k = (int)a.K;
  p.kpad = (int)round_up(a.K, 512);
  p.nc = (int)((a.K + RAW_KC - 1) / RAW_KC);
  p.corr = a.corr_mode == CORR_NONE ? 0 : 1;
  p.rt = (int)((a.N + MMQ_ROWS - 1) / MMQ_ROWS);
  const bool room = a.part && a.counter;
  const MmqPlan plan = a.passes ? MmqPlan{(int)round_up(a.pass_rows, 16), 1, MMQ_CTAS, room} : mmq_plan(a.type, a.M, a.N, a.K, room);
  p.tn = plan.tn;
  p.tt = (int)plan.tt;
  p.idesc = umma_idesc(MMQ_ROWS, p.tn > 256 ? p.tn / 2 : p.tn, bf ? 1 : 0);
  p.sa = p.tn <= 256 ? 4 : p.tn <= 320 ? 3 : 2;
  p.a_col0 = 512 - p.sa * MMQ_A_COLS;
  p.nbuf = p.tn <= 128 ? 2 : 1;
  p.status = a.status;
  p.w_wait = a.w_in_flight ? 1 : 0;
  p.passes = static_cast<const int4*>(a.passes);
  p.n_passes = a.n_passes;
  p.sorted = a.sorted;
  p.rows_out = a.passes ? (int)a.rows_out : (int)a.M;
  p.row_scale = a.row_scale;
  if (a.tp) {
    if (a.passes || a.tp->world < 1 || a.tp->world > 8 || a.N % 8 != 0 || a.tp->col_off % 8 != 0 || a.tp->ld % 8 != 0) return E_BAD_SHAPE;
    p.tp_world = a.tp->world;
    p.tp_slot = a.tp->slot;
    p.tp_col_off = a.tp->col_off;
    p.ldy = a.tp->ld;
    p.tp_epoch = a.tp->epoch;
    for (int r = 0; r < a.tp->world; ++r) {
      if (!a.tp->y_peer[r] || !a.tp->flag_peer[r] || (reinterpret_cast<uintptr_t>(a.tp->y_peer[r]) & 15)) return E_BAD_POINTER;
      p.tp_y[r] = a.tp->y_peer[r];
      p.tp_flag[r] = a.tp->flag_peer[r];
    }
  }
  // activations as [stage of 64 values][row][value]: boxes of one or two stages x tn rows, zeros beyond the matrix
  p.bg = p.tn <= 128 ? 2 : 1;
  EncodeTiledFn enc = tensor_map_encoder();
  const cuuint64_t dims[3] = {MMQ_BK, (cuuint64_t)a.M, (cuuint64_t)(a.ldb / MMQ_BK)};
  const cuuint64_t strides[2] = {(cuuint64_t)a.ldb * 2, MMQ_BK * 2};
  const cuuint32_t box[3] = {MMQ_BK, (cuuint32_t)(p.tn > 256 ? p.tn / 2 : p.tn), (cuuint32_t)p.bg};
  const cuuint32_t estr[3] = {1, 1, 1};
  if (!enc || a.ldb % MMQ_BK != 0 ||
      enc(&bmap, bf ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(a.b), dims, strides, box, estr,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return E_CUDA;
  // Shared memory: the B ring as deep as it may be (a slot is away for about 1,800 clocks between two uses: four boxes of an item of
  // 128 tokens take 2,048, four of a stage of 384 3,072), at least two raw stages, and what is left for more.
  const int corr = p.corr ? MMQ_CORR_BYTES : 0, fixed = corr + mmq_aux_bytes(a.type), b_box = p.bg * p.tn * MMQ_BK * 2;
  const int budget = 226 * 1024 - fixed, most = p.bg == 2 ? MMQ_ITEMS : MMQ_MAX_B;
  int raw = 3;
  p.sb = (budget - raw * p.raw.bytes) / b_box;
  if (p.sb < (p.bg == 2 || p.tn > 256 ? 3 : 4)) { raw = 2; p.sb = (budget - raw * p.raw.bytes) / b_box; }
  if (p.sb < 2) return E_TOO_LARGE;
  if (p.sb > most) p.sb = most;
  raw = (budget - p.sb * b_box) / p.raw.bytes;
  p.raw_stages = raw > MMQ_MAX_RAW ? MMQ_MAX_RAW : raw;
  p.corr_off = p.sb * b_box;                      // (multiples of 2,048: the tensor core reads tiles there)
  p.raw_off = p.corr_off + corr;
  p.aux_off = p.raw_off + p.raw_stages * p.raw.bytes;
  const size_t smem = 1024 + (size_t)p.aux_off + mmq_aux_bytes(a.type);
  const int64_t tiles = a.passes ? a.max_passes * p.rt : p.rt * plan.tt;
  if (tiles * p.nc * (MMQ_CTAS + 1) >= (int64_t)1 << 31) return E_TOO_LARGE;
  if (plan.shared && a.part_bytes >= 2 * plan.grid * MMQ_ROWS * p.tn * 4) {
    p.part = static_cast<float*>(a.part);
    p.counter = a.counter;
  }
  // The number of passes of a MoE step is known on the device only: there tiles are shared where that saves more than it costs.
  p.waste = a.passes ? (int)((6000 + 45 * p.tn) / (4 * mmq_stage_clocks(a.type, p.tn))) : 0;
  if (p.part && a.zero_counters > 0) {
    const int rc = launch_zero(a.counter, a.zero_counters, stream);
    if (rc) return rc;
  }
  switch (a.type) {
#define MMQ_CASE(TYPE) case TYPE: return mmq_launch<TYPE>(p, bmap, wmap, a.b_dtype, fast, (int)plan.grid, smem, stream);
    MMQ_TYPES(MMQ_CASE)
  }
  return E_BAD_TYPE;
}

}  // namespace gguf_b200
