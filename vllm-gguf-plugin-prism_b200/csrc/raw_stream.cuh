// Streaming of packed weight rows into shared memory: a stage holds 256 values (one super-block, or
// eight 32-value blocks) of each of 128 consecutive rows.  Shared by the kernels that walk 128-row
// tiles.  Three forms, chosen per matrix by plan_raw():
//
//   dense   row pitch and chunk size multiples of 16 bytes: one 2-D TMA box per stage, rows an odd number of 16-byte units apart
//   class   anything else (rows of 210, 110, 66 ... bytes): P = 16 / gcd(16, pitch) alignment classes.
//           The tensor map views the matrix as rows of P weight rows (P * pitch IS a multiple of 16), so
//           the rows of one class share the remainder of their chunk starts modulo 16 and ONE box per
//           class and stage, from the chunk start rounded down to 16 bytes into padded slots, serves
//           128 / P of them.  The N mod P rows the map cannot cover (at most seven, in the last tile)
//           arrive by one bulk copy each, in slots of their own behind the tile's 128.
//   rows    one bulk copy per row (a copy costs about 90 clocks of the SM's copy engine: only for
//           matrices that the other two cannot describe)
//
// Slots are an odd number of 16-byte units, so that eight rows read at
// the same offset fall into different banks.  Nothing is read past the caller's buffer.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace gguf_b200 {

constexpr int RAW_ROWS = 128;
constexpr int RAW_KC = 256;      // values of a row per stage
constexpr int RAW_EXTRA = 7;     // slots for rows beyond the class map

struct RawPlan {
  int mode;                // 0 rows, 1 dense, 2 class
  int cl2;                 // log2 of the number of alignment classes
  int slot;                // bytes between the rows of a stage
  int rbc;                 // bytes of a row's chunk
  int bytes;               // bytes of a stage
  int nrows, nfull;        // rows of a matrix, and how many of them the map covers
  int64_t pitch;           // bytes between weight rows
  int64_t row_bytes;       // bytes of a row that hold values
  int64_t gap;             // rows form: bytes between one matrix of nrows rows and the next
};

__device__ __forceinline__ void raw_tma_box(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_box3(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Offset, inside a stage, of row r of the tile that starts at row n0 of the matrix (whose first row is row `row0` of all
// matrices): where its slot starts, and by how much its chunk c is displaced in it.
__device__ __forceinline__ uint32_t raw_slot(const RawPlan& p, int r, int n0) {
  if (p.mode != 2) return (uint32_t)(r * p.slot);
  const int n = n0 + r;
  const int s = n >= p.nfull && n < p.nrows ? RAW_ROWS + (n - p.nfull) : ((r & ((1 << p.cl2) - 1)) << (7 - p.cl2)) | (r >> p.cl2);
  return (uint32_t)(s * p.slot);
}
__device__ __forceinline__ uint32_t raw_shift(const RawPlan& p, int n, int row0, int c) {
  if (p.mode == 1) return 0u;
  uint32_t at = (uint32_t)(row0 + n) * (uint32_t)p.pitch + (uint32_t)c * (uint32_t)p.rbc;
  if (p.gap != 0) at += ((uint32_t)row0 / (uint32_t)p.nrows) * (uint32_t)p.gap;
  return at & 15u;
}

// One row's chunk by a bulk copy into `dst`, from its address rounded down to 16 bytes; the bytes of the buffer's ragged end
// with plain loads.  Split in two so that the byte count is announced before the copy starts.
struct RawCopy { int64_t beg; uint32_t bytes; };
__device__ __forceinline__ RawCopy raw_row_copy(const RawPlan& p, const uint8_t* w, int64_t w_bytes, int64_t row, int c, uint8_t* dst) {
  const int64_t beg = row + (int64_t)c * p.rbc;
  const int64_t row_end = row + p.row_bytes;
  const int64_t end = beg + p.rbc < row_end ? beg + p.rbc : row_end;
  const int64_t safe = w_bytes & ~int64_t(15), a0 = beg & ~int64_t(15);
  int64_t a1 = (end + 15) & ~int64_t(15);
  if (a1 > safe) {
    for (int64_t o = safe > a0 ? safe : a0; o < end; ++o) dst[o - a0] = w[o];
    a1 = safe;
  }
  return {a0, a1 > a0 ? (uint32_t)(a1 - a0) : 0u};
}

// Chunk c of the tile of rows n0 .. n0 + 127 of the matrix whose first row is row `row0` of all matrices (w, w_bytes: all of
// them) into `stage`.  Called by a whole warp.  Announces `extra` bytes more, for copies the caller issues on the same barrier afterwards.
__device__ __forceinline__ void raw_issue(const RawPlan& p, const CUtensorMap* map, const uint8_t* w, int64_t w_bytes, int row0, int n0, int c,
                                          uint8_t* stage, uint64_t* bar, uint32_t extra, int lane) {
  if (p.mode == 1) {
    if (lane == 0) {
      mbar_expect_tx(bar, (uint32_t)(RAW_ROWS * p.slot) + extra);
      raw_tma_box(stage, map, c * (p.rbc / 4), row0 + n0, bar);
    }
    return;
  }
  if (p.mode == 2) {
    uint32_t total = (uint32_t)(RAW_ROWS * p.slot) + extra;
    RawCopy rc{0, 0u};
    const bool tail = n0 + RAW_ROWS > p.nfull && p.nfull < p.nrows;
    if (tail) {
      const int n = p.nfull + lane;
      if (n < p.nrows) rc = raw_row_copy(p, w, w_bytes, ((int64_t)row0 + n) * p.pitch, c, stage + (size_t)(RAW_ROWS + lane) * p.slot);
      uint32_t sum = rc.bytes;
#pragma unroll
      for (int m = 1; m < 8; m <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);   // (the tail has at most seven rows: lanes 0..7)
      total += __shfl_sync(0xffffffffu, sum, 0);
      __syncwarp();
    }
    if (lane == 0) {
      mbar_expect_tx(bar, total);
      for (int k = 0; k < (1 << p.cl2); ++k) {
        const int64_t off = (int64_t)k * p.pitch + (int64_t)c * p.rbc;
        raw_tma_box(stage + (size_t)k * (RAW_ROWS >> p.cl2) * p.slot, map, (int)((off & ~int64_t(15)) >> 2), (row0 + n0) >> p.cl2, bar);
      }
    }
    if (tail) {
      __syncwarp();
      if (rc.bytes) bulk_g2s(stage + (size_t)(RAW_ROWS + lane) * p.slot, w + rc.beg, rc.bytes, bar);
    }
    return;
  }
  RawCopy rc[4];
  uint32_t total = 0;
  int64_t row = ((int64_t)row0 + n0 + lane) * p.pitch;
  if (p.gap != 0) row += (int64_t)((unsigned)row0 / (unsigned)p.nrows) * p.gap;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = lane + 32 * q;
    rc[q] = n0 + r < p.nrows ? raw_row_copy(p, w, w_bytes, row + 32 * q * p.pitch, c, stage + (size_t)r * p.slot) : RawCopy{0, 0u};
    total += rc[q].bytes;
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) total += __shfl_xor_sync(0xffffffffu, total, m);
  __syncwarp();   // the plain stores of every lane are before lane 0's arrival
  if (lane == 0) {
    if (total + extra) mbar_expect_tx(bar, total + extra);
    else mbar_arrive(bar);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (rc[q].bytes) bulk_g2s(stage + (size_t)(lane + 32 * q) * p.slot, w + rc[q].beg, rc[q].bytes, bar);
}

// Byte alignment that the decoders of a type assume of every block (16-byte header loads and the like)
inline int raw_type_align(int type) {
  switch (type) {
    case T_Q4_K: case T_Q5_K: return 16;
    case T_IQ4_XS: case T_Q5_1: case T_IQ1_M: return 8;
    case T_Q4_1: case T_Q2_K: return 4;
  }
  return 2;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn tensor_map_encoder();

// Host: whether a matrix takes the dense form; the plan and (dense, class) the tensor map of a matrix of n_rows rows, `copies` such matrices (experts), `gap` bytes apart.
// False when the layout is outside what the decoders can read.
bool raw_dense(int type, int64_t K, int64_t pitch);
bool plan_raw(int type, const void* w, int64_t n_rows, int64_t copies, int64_t K, int64_t pitch, RawPlan& p, CUtensorMap& map, int64_t gap = 0);

}  // namespace gguf_b200
