// Kernel of the tensor-core GEMM (see mmq.cu); instantiated by mmq_inst_*.cu.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "kernels.h"
#include "mmq_decode.cuh"
#include "raw_stream.cuh"

namespace gguf_b200 {

constexpr int MMQ_ROWS = 128;
constexpr int MMQ_BK = 64;                           // values per stage (128 bytes of activations: one swizzle row)
constexpr int MMQ_GROUPS = 4;                        // producer groups of 128 threads, one thread per weight row
constexpr int MMQ_PRODUCER_WARPS = 4 * MMQ_GROUPS;
constexpr int MMQ_THREADS = (MMQ_PRODUCER_WARPS + 3) * 32;   // + B loader, MMA issuer, raw-weight loader
// Operand A moves in items: half a 256-value chunk, two stages, 64 columns of tensor memory.  Up to 256 tokens a tile there are 256
// columns of accumulator -- two of 128 tokens, or one beyond 128 -- and four A slots; up to 320 tokens, one accumulator and three A slots,
// up to 384, two.  The items' barriers are a ring of four in all cases: a group's items are four apart, so by the time it
// waits for a phase it has seen the one before complete.
constexpr int MMQ_A_COLS = 64, MMQ_ITEMS = 4, MMQ_D_STEP = 128;
constexpr int MMQ_MAX_B = 8;
// Activations arrive a box at a time, one stage or -- up to 128 tokens a tile, where the stages are short -- one item.
constexpr int MMQ_MAX_RAW = 8;
// Correction values of a block of four chunks: 32 fp16 per row, half of a tile of operand A in shared memory (K-major, 128-byte
// swizzle); the next block's go into the other half.  (Whole tiles of eight chunks, twice, took 16 KB more: at 256 tokens a tile that is the
// fifth slot of the activation ring.)
constexpr int MMQ_CORR_CHUNKS = 4, MMQ_CORR_BYTES = MMQ_ROWS * 128;

struct MmqParams {
  RawPlan raw;
  const uint8_t* w;
  int64_t w_bytes;
  void* y;
  int64_t ldy;
  int dtype;              // of y
  int n, m;               // weight rows, tokens
  int k, kpad;
  int nc, corr;           // 256-value chunks of a row; 1: half a stage of corrections behind every four of them
  int rt, tt, tn;         // row tiles, token tiles, tokens per tile (a multiple of 16, at most 256, or of 32, at most 384)
  int sa, a_col0;         // A slots: how many (2 to 4), first column
  int nbuf;               // accumulators, MMQ_D_STEP columns apart
  int bg;                 // stages of an activation box: 1 or 2
  int sb, raw_stages;     // ring depths: boxes, raw chunks
  int raw_off, aux_off, corr_off;   // shared memory behind the B ring
  uint32_t idesc;
  float* part;            // partial tiles, two slots of 128 x tn per CTA; null: every tile is one CTA's
  int w_wait;             // the weights may still be written when the kernel starts
  int waste;              // idle chunks of a CTA up to which whole tiles are dealt out all the same
  int* counter;           // arrivals per tile, zero at the start
  int* status;
  // MoE (passes != null): pass = {expert, first activation row, rows}
  const int4* passes;
  const int32_t* n_passes;
  const int32_t* sorted;  // output row of every activation row
  int rows_out;
  const float* row_scale;
  // tensor-parallel output (tp_world > 0): see MmqTp
  int tp_world, tp_slot;
  int64_t tp_col_off;
  unsigned* tp_epoch;
  void* tp_y[8];
  unsigned* tp_flag[8];
};

// ---- tcgen05 wrappers -------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// (by the lane with `lead` set, of a converged warp)
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t lead) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// one lane of a converged warp (the same one every time)
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 32 registers -> 32 consecutive columns of this thread's lane (warp w owns lanes 32 * (w % 4) ...)
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// A stage: four times D[tmem] (+)= A[tmem] * B[smem], issued by the lane with `lead` set.  16 values a time: eight columns of A (128 lanes
// x 16 fp16, two per column), 32 bytes of B = +2 in the descriptor's 16-byte units.
__device__ __forceinline__ void umma_f16_ts4(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 b0, b1, b2, b3;\n\t.reg .b32 a1, a2, a3, l1, l2, l3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {l1, %3};\n\tmov.b64 b2, {l2, %3};\n\tmov.b64 b3, {l3, %3};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %4, p;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %4, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %4, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(lead)
      : "memory");
}
// Half a stage with A from shared memory (low words of both descriptors; they share the high one)
__device__ __forceinline__ void umma_f16_ss2(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q, t;\n\t.reg .b64 a, b;\n\t.reg .b32 al, bl;\n\t"
      "setp.ne.b32 q, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, t;\n\t"
      "add.u32 al, %1, 2;\n\tadd.u32 bl, %2, 2;\n\tmov.b64 a, {al, %3};\n\tmov.b64 b, {bl, %3};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(lead)
      : "memory");
}
// K-major, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart (stride byte offset),
// leading byte offset unused by swizzled K-major layouts (1), descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16 instruction descriptor: fp32 accumulator, A/B format (0 = f16, 1 = bf16), both K-major
__host__ __device__ inline uint32_t umma_idesc(int m, int n, int fmt) {
  return (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// CTAs of the tensor-parallel launch in flight per call slot that have stored their tiles
static __device__ unsigned g_mmq_tp_done[64];

// End of a tensor-parallel launch, called by every thread of a CTA after its stores to the peers:
// CTA barrier, thread 0 fences system-wide and counts the CTA off; the last CTA of the grid
// increments this rank's launch counter and raises the slot's flag on every rank.  The flags only
// grow (one increment per rank and launch), so replays of a captured graph need no reset.
__device__ __forceinline__ void tp_finish(unsigned* epoch, unsigned* const* flag, int world, int slot, unsigned total_ctas) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    unsigned* done = &g_mmq_tp_done[slot & 63];
    const unsigned prev = atomicAdd(done, 1u);
    if (prev == total_ctas - 1) {
      *done = 0;
      __threadfence_system();
      epoch[slot] += 1;
      __threadfence_system();
      for (int r = 0; r < world; ++r) atomicAdd_system(flag[r] + slot, 1u);
    }
  }
}

// A CTA's work: a range of units (tile, chunk) in parts of one tile each.  Every role of the CTA walks the same parts.
struct MmqPart {
  int left;                  // units behind this part
  int tile, outer, inner;    // tile = outer * (row tiles of a pass, or token tiles of a row tile) + inner
  int c0, c1;                // chunks [c0, c1) of the tile
};
struct MmqTile {
  int n0;                    // first row
  int x0, rows;              // first activation row, rows that count
  int row0;                  // MoE: first row of the expert's matrix among all rows
};
// (waited: behind this thread's pdl_wait)
__device__ __forceinline__ MmqTile mmq_tile(const MmqParams& p, const MmqPart& q, bool waited) {
  MmqTile t;
  if (p.passes) {
    const int4 info = waited ? p.passes[q.outer] : ld_older(p.passes + q.outer);
    t.n0 = q.inner * MMQ_ROWS;
    t.row0 = info.x * p.n;
    t.x0 = info.y;
    t.rows = info.z;
  } else {   // token tiles of a row tile are neighbours: they share its weights in L2
    t.n0 = q.outer * MMQ_ROWS;
    t.row0 = 0;
    t.x0 = q.inner * p.tn;
    t.rows = p.m - t.x0 < p.tn ? p.m - t.x0 : p.tn;
  }
  return t;
}
// The units from u on, `units` of them, before the first part.  (The only divisions: a part behind another begins a tile.)
__device__ __forceinline__ MmqPart mmq_parts(const MmqParams& p, int u, int units) {
  const int d = p.passes ? p.rt : p.tt;
  MmqPart q;
  q.left = units;
  q.tile = (int)((unsigned)u / (unsigned)p.nc);
  q.c0 = u - q.tile * p.nc;
  q.outer = (int)((unsigned)q.tile / (unsigned)d);
  q.inner = q.tile - q.outer * d;
  q.c1 = -1;                 // (no part yet)
  return q;
}
__device__ __forceinline__ bool mmq_next_part(const MmqParams& p, MmqPart& q) {
  if (q.left <= 0) return false;
  if (q.c1 >= 0) {
    ++q.tile;
    if (++q.inner == (p.passes ? p.rt : p.tt)) { q.inner = 0; ++q.outer; }
    q.c0 = 0;
  }
  q.c1 = q.left < p.nc - q.c0 ? q.c0 + q.left : p.nc;
  q.left -= q.c1 - q.c0;
  return true;
}
// The stages of a part come in blocks: four per chunk, and behind every run of chunks with the same c / 4 half a stage of their
// correction columns (formats without them: one block).  End of the block that starts at chunk c:
__device__ __forceinline__ int mmq_block_end(const MmqParams& p, const MmqPart& q, int c) {
  const int e = (c | (MMQ_CORR_CHUNKS - 1)) + 1;
  return p.corr && e < q.c1 ? e : q.c1;
}
template <typename I, bool HAVE = I::HAVE> struct ItemStateOf { struct type {}; };
template <typename I> struct ItemStateOf<I, true> { using type = typename I::State; };
template <typename I> using ItemState = typename ItemStateOf<I>::type;

// bits of v in a 16-bit output type
__device__ __forceinline__ uint16_t mmq_bits16(int dtype, float v) {
  return dtype == DT_F16 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
// Sixteen tokens of a warp's 32 rows (a lane has one row) into this rank's column block of every rank's matrix.  What crosses
// NVLink leaves in 16-byte stores: squares of eight rows by eight tokens (fp32: four by four) are transposed across the lanes
// first, bit k of the lane against bit k of the token, so that a lane ends up with consecutive columns of one token.
// n: the lane's row; rows come in whole groups of eight.  tokens: how many of the sixteen count.  (7168 rows of
// Q4_K, 512 tokens, the matrices of 1 / 2 / 4 / 8 ranks all on one GPU: 55.7 / 57.9 / 56.8 / 61.1 us with a 2-byte store per value
// and rank, 42.4 / 44.7 / 49.4 / 59.3 so.)
__device__ __forceinline__ void mmq_store_peers(const MmqParams& p, int64_t orow, int tokens, int n, bool live, uint32_t (&acc)[16], int lane) {
  const bool f32 = p.dtype == DT_F32;
  const int group = f32 ? 4 : 8, l = lane & (group - 1);
  const int64_t at = orow * p.ldy + p.tp_col_off + (n - l);
  auto swap = [&](uint32_t& keep0, uint32_t& keep1, int bit) {   // the lane without the bit gives keep1, the one with it keep0
    const bool up = (lane & bit) != 0;
    const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? keep0 : keep1, bit);
    if (up) keep0 = got;
    else keep1 = got;
  };
#pragma unroll 1
  for (int t0 = 0; t0 < 16; t0 += group) {
    uint32_t q[4];
    if (f32) {
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = acc[i];
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        q[i] = (uint32_t)mmq_bits16(p.dtype, __uint_as_float(acc[2 * i])) | (uint32_t)mmq_bits16(p.dtype, __uint_as_float(acc[2 * i + 1])) << 16;
    }
    const int b1 = f32 ? 2 : 4, b0 = f32 ? 1 : 2;
    swap(q[0], q[2], b1);
    swap(q[1], q[3], b1);
    swap(q[0], q[1], b0);
    swap(q[2], q[3], b0);
    if (!f32) {   // the last bit: halves of a register
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, q[i], 1);
        q[i] = lane & 1 ? __byte_perm(got, q[i], 0x7632) : __byte_perm(q[i], got, 0x5410);
      }
    }
    if (live && t0 + l < tokens) {
      const int64_t e = at + (int64_t)(t0 + l) * p.ldy;
#pragma unroll 1
      for (int rk = 0; rk < p.tp_world; ++rk)
        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.tp_y[rk]) + e * (f32 ? 4 : 2)) = make_uint4(q[0], q[1], q[2], q[3]);
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) acc[i] = f32 || i >= 8 ? acc[i + 4] : acc[i + 8];   // (register indexes are static)
  }
}

// TP: the tensor-parallel form, kernels of their own.  (Sixteen-byte stores to the peers as one more branch of the same epilogue
// cost calls that never take it: 300 tokens of 8192x28672 IQ3_S 133 -> 139 us.)
template <int TYPE, typename ab_t, bool FAST, bool TP>
__global__ void __launch_bounds__(MMQ_THREADS, 1) mmq_kernel(const __grid_constant__ CUtensorMap bmap, const __grid_constant__ CUtensorMap wmap,
                                                             const __grid_constant__ MmqParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));   // swizzle atoms
  using Dec = Decoder<TYPE, ab_t>;
  const int b_stage = p.tn * MMQ_BK * 2;
  uint8_t* sB = smem;
  uint8_t* sRaw = smem + p.raw_off;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.aux_off);
  uint64_t* full = bars;                     // [4] item i % 4: its A slot is filled (the four warps of a group), boxes of an item: and its box is there
  uint64_t* empty = bars + 4;                // [4] the MMAs that read it are done
  uint64_t* b_full = bars + 8;               // [8] a box of one stage is there; boxes of an item: [0], [1] those of the blocks' corrections, in turn
  uint64_t* b_empty = bars + 16;             // [8] ... and has been read
  uint64_t* accum = bars + 24;               // [2] an accumulator is complete
  uint64_t* drained = bars + 26;             // [2] ... and has been read
  uint64_t* raw_full = bars + 28;            // [8]
  uint64_t* raw_empty = bars + 36;           // [8] read by the two groups that decode it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 44);
  volatile int* gave_up = reinterpret_cast<volatile int*>(tmem_slot + 1);   // set by any thread whose wait ran out
  volatile int* s_flag = gave_up + 1;        // [2]: the last to arrive at the tile of the part just read out / of the CTA's first part
  uint8_t* s_tab = smem + p.aux_off + 512;   // decoder tables

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (known to be the same in a warp)
  if (threadIdx.x == 0) {
    for (int s = 0; s < MMQ_ITEMS; ++s) {
      mbar_init(&full[s], MMQ_PRODUCER_WARPS / MMQ_GROUPS + (p.bg == 2 ? 1 : 0));
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < MMQ_MAX_B; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&accum[s], 1);
      mbar_init(&drained[s], MMQ_PRODUCER_WARPS);
    }
    for (int s = 0; s < MMQ_MAX_RAW; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], MMQ_PRODUCER_WARPS / 2);
    }
    *gave_up = 0;
    fence_barrier_init();
  }
  decoder_fill_tables<TYPE, ab_t>(s_tab);
  if (warp == MMQ_PRODUCER_WARPS) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem_base = 0;   // (all 512 columns are this CTA's)
  pdl_trigger();   // the next kernel may become resident; it waits for this one before it touches anything
  // What the kernel ahead writes: the activations, and -- cleared, or read until now -- what the epilogue writes.  Everything else, decoding
  // included, starts before it is done (the weights: see pdl_wait; the work list of a MoE step is older than the quantizer's trigger).
  const bool moe = p.passes != nullptr;
  const int tiles = moe ? __shfl_sync(0xffffffffu, ld_older(p.n_passes), 0) * p.rt : p.rt * p.tt;
  // Units: (tile, chunk) where CTAs share tiles, whole tiles where they do not -- there is no room for parts, or the last wave
  // of whole tiles idles for less than sharing costs.  Every CTA in use has an equal contiguous range of them.
  const int rest = tiles % (int)gridDim.x;
  const bool split = p.part && rest != 0 && (unsigned)p.nc * (unsigned)((int)gridDim.x - rest) > (unsigned)p.waste * gridDim.x;
  const int U = split ? tiles * p.nc : tiles, G = U < (int)gridDim.x ? U : (int)gridDim.x;
  const int cta = (int)blockIdx.x, scale = split ? 1 : p.nc;
  const int u0 = cta < G ? (int)((unsigned)(cta * U) / (unsigned)G) * scale : 0;
  MmqPart q = mmq_parts(p, u0, cta < G ? (int)((unsigned)((cta + 1) * U) / (unsigned)G) * scale - u0 : 0);
  const int first_tile = q.tile;
  const uint32_t bars_s = smem_u32(bars), gave_up_s = smem_u32(const_cast<const int*>(gave_up));
  auto bar = [&](int k) { return bars_s + 8u * (uint32_t)k; };   // (the numbers are those of the list above)
  const int half_n = p.tn > 256 ? p.tn / 2 : 0;   // tokens of one instruction and of one activation box, where a tile takes two
  bool ok = true;

  if (warp < MMQ_PRODUCER_WARPS) {
    // ---------------- producers and epilogue ----------------
    // The work of a part, in order: two items per chunk (a half, 128 values, two stages).  Group g takes the items g, g + 4, ...
    // (counted over the whole life of the CTA); thread r of the group decodes row n0 + r.  Item i goes to A slot i modulo their
    // number.  The tile before is read out after every group has published its first item of the next one, so that the tensor
    // core has four items of work while the accumulator goes to memory.  What an item costs beside its decoding is kept small: one
    // wait for the raw chunk, one for the slot and one signal for 128 values, and no work list but a stride.  (Stage by stage, with
    // the correction stages dealt out among the groups, it was 130 to 165 instructions per stage of 32 rows, as many as the decoding of Q4_K.)
    const int r = threadIdx.x & 127, g = threadIdx.x >> 7;
    const DecodeCtx cx = decoder_context<TYPE>(s_tab, lane);
    const int nunits = p.k / 32;
    const uint32_t d_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t a_lane = d_lane + (uint32_t)p.a_col0;
    const uint32_t s_corr = smem_u32(smem + p.corr_off) + (uint32_t)(r * 128);
    // (After a time-out the loops run on without waiting: every barrier still gets its arrivals, the result is invalid and the
    // status word says so.)
    auto wait = [&](uint32_t b, uint32_t parity) {
      mbar_wait_or(b, parity, gave_up_s);
      __syncwarp();
    };
    // Reads out part e, the pi-th of this CTA.  Kept short: this code runs two or three times in the life of a CTA, and fetching
    // its instructions costs more than running them (unrolled over an accumulator held in 64 registers it took 10,000 clocks
    // instead of 4,000, most of them for the first time through).  FINISH: the parts of e's tile are all in memory.
    enum : int { MORE, FINAL, FINISH };
    auto epilogue = [&](const MmqPart& e, int pi, int mode) {
      pdl_wait();
      const MmqTile et = mmq_tile(p, e, true);
      const int buf = p.nbuf == 2 ? pi & 1 : 0, use = p.nbuf == 2 ? pi >> 1 : pi;
      const int n = et.n0 + r, nb = p.tn / 16;
      const bool live = n < p.n;
      const bool shared = e.c1 - e.c0 < p.nc;
      // output rows (negative: none) and their weights, of the tokens this group reads: lanes 0..15 of each block of 16
      auto out_row = [&](int b) {
        const int t = 16 * b + (lane & 15);
        int o = b < nb && t < et.rows ? et.x0 + t : -1;
        if (moe && o >= 0) o = p.sorted[o];
        return o < p.rows_out ? o : -1;
      };
      auto out_scale = [&](int o) { return p.row_scale && o >= 0 ? p.row_scale[o] : 1.f; };
      int orow = out_row(g);
      float scale = out_scale(orow);
      if (mode != FINISH) {
        wait(bar(24 + buf), (uint32_t)use & 1u);
        tc_fence_after();
      }
      const uint32_t d = d_lane + (uint32_t)(buf * MMQ_D_STEP);
      int first = 0, last = 0, s_first = 0;
      bool in_tmem = mode != FINISH;
      const int slot4 = p.tn * 32;            // float4s of a partial tile
      float4* part = reinterpret_cast<float4*>(p.part) + r;
      if (shared) {
        // The CTAs first .. last share the tile.  The last of them to arrive adds the parts in CTA order (deterministic).
        const int ta = e.tile * p.nc;
        first = (int)((unsigned)((ta + 1) * G - 1) / (unsigned)U);
        last = (int)((unsigned)((ta + p.nc) * G - 1) / (unsigned)U);
        s_first = 2 * first + ((unsigned)(first * U) / (unsigned)G >= (unsigned)ta ? 0 : 1);
        if (mode != FINISH) {
          if (mode == FINAL && e.c0 == 0) {   // the others did their parts first: if all are there, this one need not be published
            if (threadIdx.x == 0) {
              int seen;
              asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.counter + e.tile) : "memory");
              s_flag[0] = seen == last - first ? 2 : 0;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(MMQ_PRODUCER_WARPS * 32) : "memory");
            in_tmem = s_flag[0] == 2;
          } else {
            in_tmem = false;
          }
          if (!in_tmem) {
            float4* out = part + (size_t)(2 * cta + (e.tile == first_tile ? 0 : 1)) * slot4;
#pragma unroll 1
            for (int b = g; b < nb; b += MMQ_GROUPS) {
              uint32_t acc[16];
              __syncwarp();
              tmem_ld16(d + (uint32_t)(16 * b), acc);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 4; ++j)
                __stcg(out + (4 * b + j) * 128, make_float4(__uint_as_float(acc[4 * j]), __uint_as_float(acc[4 * j + 1]),
                                                            __uint_as_float(acc[4 * j + 2]), __uint_as_float(acc[4 * j + 3])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&drained[buf]);
            asm volatile("bar.sync 1, %0;" ::"n"(MMQ_PRODUCER_WARPS * 32) : "memory");
            if (threadIdx.x == 0) {
              __threadfence();   // cumulative: covers what the barrier made visible to this thread
              s_flag[mode == MORE ? 1 : 0] = atomicAdd(p.counter + e.tile, 1) == last - first ? 1 : 0;
              __threadfence();
            }
            if (mode == MORE) return;
            asm volatile("bar.sync 1, %0;" ::"n"(MMQ_PRODUCER_WARPS * 32) : "memory");
            if (s_flag[0] == 0) return;
          }
        }
      }
      const bool plain = !TP && p.dtype != DT_F32, rows = plain && !moe && !p.row_scale;
#pragma unroll 1
      for (int b = g; b < nb; b += MMQ_GROUPS) {
        const int orow_next = out_row(b + MMQ_GROUPS);
        uint32_t acc[16];
        if (in_tmem) {
          __syncwarp();
          tmem_ld16(d + (uint32_t)(16 * b), acc);
          tmem_ld_wait();
        }
        if (shared) {
          if (!in_tmem) {   // (in tensor memory: only ever the part of the first CTA of the tile)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] = 0u;
          }
#pragma unroll 2
          for (int c = in_tmem ? first + 1 : first; c <= last; ++c) {
            const float4* in = part + (size_t)(c == first ? s_first : 2 * c) * slot4 + 4 * b * 128;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float4 v = __ldcg(in + j * 128);
              acc[4 * j] = __float_as_uint(__uint_as_float(acc[4 * j]) + v.x);
              acc[4 * j + 1] = __float_as_uint(__uint_as_float(acc[4 * j + 1]) + v.y);
              acc[4 * j + 2] = __float_as_uint(__uint_as_float(acc[4 * j + 2]) + v.z);
              acc[4 * j + 3] = __float_as_uint(__uint_as_float(acc[4 * j + 3]) + v.w);
            }
          }
        }
        if (rows) {   // consecutive rows: 5 instructions a value (20 through the row numbers, a tenth of all the kernel issued at 512 tokens)
          uint32_t h[8];
          if (p.dtype == DT_F16) {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2<__half>(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2<__nv_bfloat16>(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
          }
          const int left = live ? et.rows - 16 * b : 0;
          uint16_t* y = static_cast<uint16_t*>(p.y) + (int64_t)(et.x0 + 16 * b) * p.ldy + n;
          if (left >= 16) {
#pragma unroll
            for (int j = 0; j < 16; ++j, y += p.ldy) *y = (uint16_t)(j & 1 ? h[j >> 1] >> 16 : h[j >> 1]);
          } else {
#pragma unroll 1
            for (int j = 0; j < left; ++j, y += p.ldy) {
              *y = (uint16_t)h[0];
              h[0] = __funnelshift_r(h[0], h[1], 16);
#pragma unroll
              for (int i = 1; i < 7; ++i) h[i] = __funnelshift_r(h[i], h[i + 1], 16);
              h[7] >>= 16;
            }
          }
        } else if (plain) {   // rows of their own: lane j of each sixteen has the number and the weight of row j
          uint32_t h[8];
          if (p.dtype == DT_F16) {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2<__half>(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = pack2<__nv_bfloat16>(__uint_as_float(acc[2 * j]), __uint_as_float(acc[2 * j + 1]));
          }
          if (p.row_scale) {   // applied as the reference applies it: to the rounded value, rounded again
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float s0 = __shfl_sync(0xffffffffu, scale, 2 * j), s1 = __shfl_sync(0xffffffffu, scale, 2 * j + 1);
              if (p.dtype == DT_F16) {
                const float2 f = __half22float2(u32_as_h2(h[j]));
                h[j] = pack2<__half>(f.x * s0, f.y * s1);
              } else {
                h[j] = pack2<__nv_bfloat16>(__uint_as_float(h[j] << 16) * s0, __uint_as_float(h[j] & 0xFFFF0000u) * s1);
              }
            }
          }
          uint8_t* y = static_cast<uint8_t*>(p.y) + 2 * (int64_t)n;
          const uint32_t pitch = 2u * (uint32_t)p.ldy;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int o = __shfl_sync(0xffffffffu, orow, j);
            if (live && o >= 0) *reinterpret_cast<uint16_t*>(y + (uint64_t)(uint32_t)o * pitch) = (uint16_t)(j & 1 ? h[j >> 1] >> 16 : h[j >> 1]);
          }
        } else if constexpr (TP) {
          mmq_store_peers(p, et.x0 + 16 * b, et.rows - 16 * b, n, live, acc, lane);
        } else {
#pragma unroll 1
          for (int j = 0; j < 16; ++j) {
            const int o = __shfl_sync(0xffffffffu, orow, j);
            const float w = __shfl_sync(0xffffffffu, scale, j), v = __uint_as_float(acc[0]);
            if (live && o >= 0) static_cast<float*>(p.y)[(int64_t)o * p.ldy + n] = p.row_scale ? v * w : v;
#pragma unroll
            for (int k = 0; k < 15; ++k) acc[k] = acc[k + 1];   // (register indexes are static)
          }
        }
        orow = orow_next;
        scale = out_scale(orow);
      }
      if (in_tmem) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&drained[buf]);
      }
    };

    // Item i is half i & 1 of the i / 2-th chunk of the CTA, so a group has the same half, slot and barriers all its life.
    const int half = g & 1;
    const bool wide = p.raw.mode == 1 || (p.raw.mode == 2 && p.raw.cl2 == 0);   // rows of one remainder modulo 16
    const uint32_t slot_free = bar(4 + ((g - p.sa) & 3));          // `empty` of the item that had the slot before
    uint32_t free_ph = g >= p.sa ? 0u : 1u;                        // (1 at first: the slot has never been used)
    int a_slot = g >= p.sa ? g - p.sa : g;                         // (four items on: the next slot of three, the same of two or four)
    int rs = g >> 1;             // raw slot of the group's next chunk, and its phase
    uint32_t rph = 0;
    int i0 = 0, pi = 0;          // items before the part, parts so far
    int blk0 = 0, end2 = -1;     // blocks of corrections before the part; last item of the last but one of them
    MmqPart prev{}, head{};      // the part before, the CTA's first part
    int mode = MORE;
    for (;;) {
      const bool more = mode == MORE && mmq_next_part(p, q);
      if (!more && mode == MORE) mode = FINAL;
      const bool waited = pi > 0;
      if (moe && waited) pdl_wait();   // (over: the part before has had its activations)
      const MmqTile qt = mmq_tile(p, q, waited);
      const int n = qt.n0 + r;
      const uint8_t* slot = sRaw + raw_slot(p.raw, r, qt.n0);
      const int items = more ? 2 * (q.c1 - q.c0) : 0;
      int m = (g - i0) & 3;      // this group's next item of the part
      bool read_out = pi > 0;
      // With one accumulator and fewer slots than groups the first items of the last groups have no room before the tile is read out.
      bool hold = read_out && p.nbuf == 1 && m >= p.sa;
      for (;;) {
        if (m < items && !hold) {
          const int c = q.c0 + (m >> 1), i = i0 + m;
          // The group has seen the chunk before the last one land; with three slots that does not tell that this slot's last chunk has,
          // and a wait that is a phase early returns at once.
          if (p.raw_stages == 3) wait(bar(36 + rs), rph ^ 1u);
          wait(bar(28 + rs), rph);
          const uint8_t* chunk = slot + rs * p.raw.bytes + (FAST ? 0u : raw_shift(p.raw, n, qt.row0, c));
          uint2 cv;
          if constexpr (Dec::CORR) cv = Dec::corr(chunk, half, nunits - 8 * c);
          using Item = Item128<TYPE, ab_t>;
          ItemState<Item> state;
          const uint32_t row_s = smem_u32(chunk);
          if constexpr (Item::HAVE) Item::begin(row_s, half, wide, nunits - 8 * c - 4 * half, state);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int s2 = 2 * half + h;      // 64-value stage of the chunk
            uint32_t v[32];
            if constexpr (Item::HAVE) {
              if (h == 0) Item::template stage<0>(row_s, half, wide, cx, state, v);
              else Item::template stage<1>(row_s, half, wide, cx, state, v);
            } else if constexpr (FAST) {
              Stage64<TYPE, ab_t>::decode(chunk, s2, v);
            } else {
              const int u = 2 * s2;           // units (32 values) u, u + 1 of the chunk
              // (rows beyond the matrix decode what their slots happen to hold: nothing reads their sums)
              const int left = BlockTraits<TYPE>::QK == 256 ? 2 : nunits - 8 * c - u;
              uint32_t (&v0)[16] = *reinterpret_cast<uint32_t (*)[16]>(&v[0]);
              uint32_t (&v1)[16] = *reinterpret_cast<uint32_t (*)[16]>(&v[16]);
              uint32_t raw[Dec::RW];
              if (left > 0) {
                Dec::load(chunk, u, raw);
                Dec::decode(chunk, u, raw, cx, v0);
              } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v0[j] = 0;
              }
              if (left > 1) {
                if constexpr (!decoder_pair_load<TYPE>()) Dec::load(chunk, u + 1, raw);   // (one load serves both)
                Dec::decode(chunk, u + 1, raw, cx, v1);
              } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v1[j] = 0;
              }
            }
            if (h == 1) {   // this warp is done reading the raw chunk: hand the slot back to the loader
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(36 + rs));
            } else {
              wait(slot_free, free_ph);
              free_ph ^= 1u;
              tc_fence_after();
            }
            tmem_st32(a_lane + (uint32_t)(a_slot * MMQ_A_COLS + 32 * h), v);
          }
          if constexpr (Dec::CORR) {
            // The block's half tile: multiplied before the last item of the block is handed back, and free again for the block after
            // the next.  That item is three before this one at the earliest, and four slots wait for the fourth.
            const int b = (c >> 2) - (q.c0 >> 2);
            const int piece0 = (blk0 + b) & 1 ? 4 ^ (r & 7) : r & 7;     // 16-byte piece of the block's first chunk, swizzled
            if (half == 0 && (c == q.c0 || (c & 3) == 0)) {   // the block's first item
              const int e = b == 0 ? end2 : b == 1 ? i0 - 1 : i0 + 2 * ((c & ~3) - 4 - q.c0) - 1;
              if (e >= 0 && e > i - p.sa) wait(bar(4 + (e & (MMQ_ITEMS - 1))), (uint32_t)(e >> 2) & 1u);
              const int lo = c & 3, hi = q.c1 - (c & ~3);     // chunks that other parts have, or nobody: zeros
              if (lo > 0 || hi < 4) {
#pragma unroll 1
                for (int j = 0; j < 4; ++j)
                  if (j < lo || j >= hi) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(s_corr + (uint32_t)((j ^ piece0) << 4)), "r"(0u) : "memory");
              }
            }
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(s_corr + (uint32_t)((((c & 3) ^ piece0) << 4) + 8 * half)), "r"(cv.x), "r"(cv.y) : "memory");
            fence_proxy_async();   // (the tensor core reads it)
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(g));
          m += 4;
          if (p.sa == 3) a_slot = a_slot == 2 ? 0 : a_slot + 1;
          rs += 2;
          if (rs >= p.raw_stages) { rs -= p.raw_stages; rph ^= 1u; }
        }
        if (read_out) {
          epilogue(prev, pi - 1, mode);
          read_out = false;
        }
        if (m >= items) break;
        hold = false;
      }
      i0 += items;
      if constexpr (Dec::CORR) {
        if (more) {
          const int nb = ((q.c1 - 1) >> 2) - (q.c0 >> 2) + 1;
          end2 = nb > 1 ? i0 - 2 * (q.c1 - ((q.c1 - 1) & ~3)) - 1 : i0 - items - 1;
          blk0 += nb;
        }
      }
      if (!more) {
        if (mode == FINISH || head.c1 - head.c0 == p.nc || pi < 2) break;
        asm volatile("bar.sync 1, %0;" ::"n"(MMQ_PRODUCER_WARPS * 32) : "memory");
        if (s_flag[1] == 0) break;
        mode = FINISH;           // the first part's tile fell to this CTA after all: once more, for it
        prev = head;
        continue;
      }
      if (pi == 0) head = q;
      prev = q;
      ++pi;
    }
  } else if (warp == MMQ_PRODUCER_WARPS) {
    // ---------------- B loader: one TMA box (64 or 2 x 64 values x tn rows; two beyond 256) per stage or item ----------------
    // (Converged like the MMA issuer below.)
    const uint32_t lead = elect_one() ? 1u : 0u;
    const uint32_t bytes = (uint32_t)(p.bg * b_stage), sb_s = smem_u32(sB);
    int i = 0, sb = 0, blk = 0;
    uint32_t ph = 0;
    pdl_wait();
    while (mmq_next_part(p, q)) {
      const int x0 = mmq_tile(p, q, true).x0;
      for (int cs = q.c0, ce; cs < q.c1; cs = ce, ++blk) {
        ce = mmq_block_end(p, q, cs);
        const int n = 2 * (ce - cs) * (p.bg == 2 ? 1 : 2);
#pragma unroll 1
        for (int j = 0; j < n + p.corr; ++j) {
          mbar_wait_or(bar(16 + sb), ph ^ 1u, gave_up_s);
          if (lds32(gave_up_s) != 0u) goto b_done;   // (no copy into a slot that may be in use)
          __syncwarp();
          const int stage = j < n ? 4 * cs + p.bg * j : (p.kpad >> 6) + (cs >> 3);   // (eight chunks' columns: a block takes its half)
          const uint32_t fb = bar(p.bg == 1 ? 8 + sb : j < n ? i & (MMQ_ITEMS - 1) : 8 + (blk & 1)), dst = sb_s + (uint32_t)sb * bytes;
          if (lead) {
            mbar_expect_tx(fb, bytes);
            tma_box3(dst, &bmap, 0, x0, stage, fb);
            if (half_n) tma_box3(dst + (uint32_t)(half_n * (MMQ_BK * 2)), &bmap, 0, x0 + half_n, stage, fb);
          }
          i += j < n ? 1 : 0;
          if (++sb == p.sb) { sb = 0; ph ^= 1u; }
        }
      }
    }
  b_done:;
  } else if (warp == MMQ_PRODUCER_WARPS + 2) {
    // ---------------- raw-weight loader ----------------
    if (p.w_wait) pdl_wait();
    int st = 0;
    uint32_t sph = 0;
    while (ok && mmq_next_part(p, q)) {
      const MmqTile qt = mmq_tile(p, q, false);
      for (int c = q.c0; c < q.c1; ++c) {
        mbar_wait_or(bar(36 + st), sph ^ 1u, gave_up_s);
        if (lds32(gave_up_s) != 0u) { ok = false; break; }
        __syncwarp();
        raw_issue(p.raw, &wmap, p.w, p.w_bytes, qt.row0, qt.n0, c, sRaw + (size_t)st * p.raw.bytes, &raw_full[st], 0u, lane);
        __syncwarp();
        if (++st == p.raw_stages) { st = 0; sph ^= 1u; }
      }
    }
  } else {
    // ---------------- MMA issuer ----------------
    // The warp stays converged and its control flow depends on nothing but parameters, so that addresses, descriptors and counters
    // live in uniform registers; one lane issues.  (With one lane in the loop, every operand went from a register to a uniform one at
    // each instruction, and this loop was what bounded the kernel at 128 tokens or less: 460 to 560 clocks a stage whatever the decoder.)
    const uint32_t lead = elect_one() ? 1u : 0u;
    int i = 0, sb = 0, pi = 0, blk = 0, a_slot = 0;
    uint32_t ph = 0;
    const uint64_t bd0 = umma_desc_sw128(smem_u32(sB));
    const uint32_t b_step = (uint32_t)(b_stage >> 4), b_lo0 = (uint32_t)bd0, b_hi = (uint32_t)(bd0 >> 32);
    const uint32_t c_lo0 = (uint32_t)umma_desc_sw128(smem_u32(smem + p.corr_off));
    const uint32_t half_lo = (uint32_t)(half_n * (MMQ_BK * 2) >> 4);
    uint32_t b_lo = b_lo0;
    auto box_done = [&]() {   // the box just multiplied goes back
      umma_commit(bar(16 + sb), lead);
      b_lo += (uint32_t)p.bg * b_step;
      if (++sb == p.sb) { sb = 0; ph ^= 1u; b_lo = b_lo0; }
    };
    while (mmq_next_part(p, q)) {
      const int buf = p.nbuf == 2 ? pi & 1 : 0, use = p.nbuf == 2 ? pi >> 1 : pi;
      mbar_wait_or(bar(26 + buf), ((uint32_t)use & 1u) ^ 1u, gave_up_s);
      const uint32_t d = (uint32_t)(buf * MMQ_D_STEP);
      uint32_t accumulate = 0;
      for (int cs = q.c0, ce; cs < q.c1; cs = ce) {
        ce = mmq_block_end(p, q, cs);
#pragma unroll 1
        for (int end = i + 2 * (ce - cs); i < end; ++i) {
          const int s = i & (MMQ_ITEMS - 1);
          mbar_wait_or(bar(s), (uint32_t)(i >> 2) & 1u, gave_up_s);
          const uint32_t at = (uint32_t)(p.a_col0 + a_slot * MMQ_A_COLS);
          if (++a_slot == p.sa) a_slot = 0;
          if (p.bg == 2) {
            __syncwarp();
            tc_fence_after();
            umma_f16_ts4(d, at, b_lo, b_hi, p.idesc, accumulate, lead);
            umma_f16_ts4(d, at + 32, b_lo + b_step, b_hi, p.idesc, 1u, lead);
            box_done();
          } else {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              mbar_wait_or(bar(8 + sb), ph, gave_up_s);
              __syncwarp();
              tc_fence_after();
              umma_f16_ts4(d, at + 32 * h, b_lo, b_hi, p.idesc, accumulate | (uint32_t)h, lead);
              if (half_n) umma_f16_ts4(d + (uint32_t)half_n, at + 32 * h, b_lo + half_lo, b_hi, p.idesc, accumulate | (uint32_t)h, lead);
              box_done();
            }
          }
          accumulate = 1;
          if (p.corr && i == end - 1) {   // the block's corrections, before its last item is handed back
            mbar_wait_or(bar(8 + (p.bg == 2 ? blk & 1 : sb)), p.bg == 2 ? (uint32_t)(blk >> 1) & 1u : ph, gave_up_s);
            __syncwarp();
            tc_fence_after();
            const uint32_t c_lo = c_lo0 + 4u * (uint32_t)(blk & 1), x_lo = b_lo + 4u * (uint32_t)((cs >> 2) & 1);   // halves of 64 bytes
            umma_f16_ss2(d, c_lo, x_lo, b_hi, p.idesc, lead);
            if (half_n) umma_f16_ss2(d + (uint32_t)half_n, c_lo, x_lo + half_lo, b_hi, p.idesc, lead);
            ++blk;
            box_done();
          }
          umma_commit(bar(4 + s), lead);
        }
      }
      umma_commit(bar(24 + buf), lead);   // completes once every tcgen05.mma issued so far has finished
      ++pi;
    }
    __syncwarp();
  }
  if (!ok) *gave_up = 1;   // (any lane)
  tc_fence_before();
  __syncthreads();
  if (*gave_up) {
    if (threadIdx.x == 0) atomicExch(p.status, E_TIMEOUT);
    // A bounded wait ran out somewhere in this CTA (the result is invalid and the status word says so).  Before the tensor
    // memory is released and the CTA retires, everything it started must have finished: the commit below covers the tensor
    // pipe (bounded wait on a barrier nobody else uses any more), and the copies still in flight depend on nothing and land
    // within microseconds, so a pause far longer than their latency covers them.  Nothing here can wait for ever.
    if (warp == MMQ_PRODUCER_WARPS + 1) {
      uint64_t* end = bars + 48;
      if (lane == 0) mbar_init(end, 1);
      __syncwarp();
      if (elect_one()) umma_commit(end);
      __syncwarp();
      mbar_wait_bounded(end, 0);
    }
    drain_pause();
    tc_fence_before();
    __syncthreads();
  }
  if (warp == MMQ_PRODUCER_WARPS) tmem_dealloc(tmem_base, 512);
  if constexpr (TP) tp_finish(p.tp_epoch, p.tp_flag, p.tp_world, p.tp_slot, gridDim.x);
}

template <int TYPE, typename ab_t, bool FAST, bool TP>
static int mmq_launch_kernel(const MmqParams& p, const CUtensorMap& bmap, const CUtensorMap& wmap, int grid, size_t smem, cudaStream_t stream) {
  auto kern = mmq_kernel<TYPE, ab_t, FAST, TP>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return E_CUDA;
    configured[dev & 63] = true;
  }
  return launch_pdl(kern, dim3((unsigned)grid), dim3(MMQ_THREADS), smem, stream, bmap, wmap, p) == cudaSuccess ? E_OK : E_CUDA;
}
template <int TYPE, typename ab_t, bool FAST>
static int mmq_launch_form(const MmqParams& p, const CUtensorMap& bmap, const CUtensorMap& wmap, int grid, size_t smem, cudaStream_t stream) {
  return p.tp_world > 0 ? mmq_launch_kernel<TYPE, ab_t, FAST, true>(p, bmap, wmap, grid, smem, stream)
                        : mmq_launch_kernel<TYPE, ab_t, FAST, false>(p, bmap, wmap, grid, smem, stream);
}
// ab: element type of the activation matrix (DT_F16, DT_BF16); fast: whole-stage decoder on dense boxes
template <int TYPE> int mmq_launch(const MmqParams& p, const CUtensorMap& bmap, const CUtensorMap& wmap, int ab, bool fast, int grid, size_t smem,
                                   cudaStream_t stream) {
  if constexpr (Stage64<TYPE, __half>::FAST) {
    if (fast) return ab == DT_F16 ? mmq_launch_form<TYPE, __half, true>(p, bmap, wmap, grid, smem, stream) : E_BAD_DTYPE;
  }
  if (fast) return E_BAD_SHAPE;
  if constexpr (decoder_bf16<TYPE>()) {
    if (ab == DT_BF16) return mmq_launch_form<TYPE, __nv_bfloat16, false>(p, bmap, wmap, grid, smem, stream);
  }
  return ab == DT_F16 ? mmq_launch_form<TYPE, __half, false>(p, bmap, wmap, grid, smem, stream) : E_BAD_DTYPE;
}
}  // namespace gguf_b200
