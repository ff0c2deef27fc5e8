// Weight decoders of the tensor-core GEMM (mmq.cu): one 32-value group of one weight row
// ("unit" u = values 32u..32u+31) -> 16 packed 16-bit pairs = 64 bytes of the row in the A tile.
// A producer thread owns one row of a 64-value stage and calls a decoder for its two units; towards the end of this file,
// whole-stage decoders replace that for Q4_K / Q5_K / Q4_0 / Q8_0 in dense stages, and decoders of an item (two stages) for Q6_K,
// IQ2_*, IQ3_*, IQ4_NL and, with fp16 activations, IQ4_XS.
//
// Each decoder is split in two:
//   load()   fetches a unit's raw bytes (from the shared-memory raw ring) into registers,
//   decode() turns those registers into fp16/bf16 values.
//
// Values are bit-identical to the reference's standalone dequantize for the types that are fed
// to the MMA as dequantized weights (Q4_0, Q8_0, Q6_K: dequantize.cuh:3-15, 69-78, 232-256;
// IQ2_XXS: dequantize.cuh:258-275), and so are the IQ3 and IQ4 values (of the split scales of fp16 every
// finite scale, sub-scale and level was compared).  Q4_K feeds half(d*sc*q) and carries its min term in
// the correction columns (see mmq.cu).
//
// Blocks of Q4_0 / Q8_0 / Q6_K / IQ2_XXS are only 2-byte aligned: raw bytes are fetched as the
// aligned 32-bit words that cover them and realigned with funnel shifts.
#pragma once

#include "common.cuh"
#include "tables.cuh"

namespace gguf_b200 {

template <typename ab_t> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {   // one instruction for both roundings
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
// (1024 + a, 1024 + b) as half2 for small unsigned a, b: exact integers, so subtracting
// 1024 + bias afterwards yields (a - bias, b - bias) without any rounding.
__device__ __forceinline__ __half2 ints_plus_1024(uint32_t a, uint32_t b) { return u32_as_h2(0x64006400u | a | (b << 16)); }
__device__ __forceinline__ __half2 hmul2_rn(__half2 a, __half2 b) { return __hmul2_rn(a, b); }
__device__ __forceinline__ uint32_t ldg16(const uint8_t* p) { return __ldg(reinterpret_cast<const uint16_t*>(p)); }

// N aligned words covering `len` bytes from the (2-byte aligned) address p in the shared-memory
// staging area of the raw weight bytes; words that hold no needed byte are not loaded.  The loads
// are explicit shared-window loads: rounding the address down through an integer made the
// compiler forget the address space, and generic loads of shared memory travel the global-memory
// pipeline (ncu: `lg_throttle` and `long_scoreboard` stalls in the decode warps).
template <int N> __device__ __forceinline__ void ldg_cover(const uint8_t* p, int len, uint32_t* r) {
  const uint32_t a = smem_u32(p);
  const uint32_t al = a & ~3u;
  const int need = (len + (int)(a & 3u) + 3) >> 2;
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = i < need ? lds32(al + 4u * i) : 0u;
}
// word i of the byte stream that starts `sh` bits into r[0]
__device__ __forceinline__ uint32_t word_at(const uint32_t* r, int i, uint32_t sh) { return __funnelshift_r(r[i], r[i + 1], sh); }
__device__ __forceinline__ uint32_t shift_of(const uint8_t* p) { return (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3) * 8u; }

// Tables in shared memory, held as 32-bit shared-window addresses so that every look-up is an
// ld.shared (through a generic pointer the look-ups travel the global-memory pipeline).  The
// look-ups are plain (non-volatile) asm: their index comes from weight bytes that are read long
// after the barrier that published the tables.
// A table is replicated, entry i of copy c at index copies * i + c, and a thread reads copy (lane mod copies): the lanes
// that share a 128-byte access phase then sit in different columns of the 128 bytes whatever entries they look up (random
// look-ups into a single copy averaged 2.5 to 3 bank conflicts per access).  The addresses below already point at this
// thread's copy; the larger code books have room for fewer copies.
// IQ3_XXS has 16 copies of the signs, of which half a warp's share a bank: with 32 the tables left two activation boxes at 384 tokens a
// tile and two raw stages at 256.  14336x4096, 32 -> 16 copies: 384 tokens 43.5 -> 41.0 us, 256 tokens 31.4 -> 29.9, 128 tokens 24.2 -> 24.4.
struct DecodeCtx {
  uint32_t grid;      // code book: byte-permute selectors of value pairs (IQ2), magnitudes (IQ3), codes (IQ1)
  uint32_t sgn;       // per 7-bit sign index, the signs of the four value pairs (iq_pair_signs)
};
template <int TYPE> struct DecodeTables {   // GRID entries of GB bytes in GC copies; SGN sign words in SC copies
  static constexpr int GRID = 0, GB = 0, GC = 0, SGN = 0, SC = 0;
};
template <> struct DecodeTables<T_IQ2_XXS> { static constexpr int GRID = 256, GB = 16, GC = 8, SGN = 128, SC = 32; };
template <> struct DecodeTables<T_IQ2_XS> { static constexpr int GRID = 512, GB = 16, GC = 4, SGN = 128, SC = 32; };
template <> struct DecodeTables<T_IQ2_S> { static constexpr int GRID = 1024, GB = 16, GC = 2, SGN = 0, SC = 0; };
template <> struct DecodeTables<T_IQ3_XXS> { static constexpr int GRID = 256, GB = 8, GC = 16, SGN = 128, SC = 16; };
template <> struct DecodeTables<T_IQ3_S> { static constexpr int GRID = 512, GB = 8, GC = 8, SGN = 0, SC = 0; };
template <> struct DecodeTables<T_IQ1_S> { static constexpr int GRID = 2048, GB = 4, GC = 2, SGN = 0, SC = 0; };
template <> struct DecodeTables<T_IQ1_M> : DecodeTables<T_IQ1_S> {};
template <int TYPE> __host__ __device__ constexpr int decoder_table_bytes() {
  using D = DecodeTables<TYPE>;
  return D::GRID * D::GB * D::GC + D::SGN * 4 * D::SC;
}
template <int TYPE> __device__ __forceinline__ DecodeCtx decoder_context(const uint8_t* tab, int lane) {
  using D = DecodeTables<TYPE>;
  DecodeCtx cx{0, 0};
  if constexpr (D::GRID > 0) cx.grid = smem_u32(tab) + (uint32_t)(D::GB * (lane & (D::GC - 1)));
  if constexpr (D::SGN > 0) cx.sgn = smem_u32(tab) + (uint32_t)(D::GRID * D::GB * D::GC + 4 * (lane & (D::SC - 1)));
  return cx;
}
template <int TYPE> __device__ __forceinline__ uint4 grid128(const DecodeCtx& cx, uint32_t i) {
  uint4 v;
  asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(cx.grid + (uint32_t)(16 * DecodeTables<TYPE>::GC) * i));
  return v;
}
template <int TYPE> __device__ __forceinline__ uint2 grid64(const DecodeCtx& cx, uint32_t i) {
  uint2 v;
  asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(cx.grid + (uint32_t)(8 * DecodeTables<TYPE>::GC) * i));
  return v;
}
template <int TYPE> __device__ __forceinline__ uint32_t grid32(const DecodeCtx& cx, uint32_t i) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(cx.grid + (uint32_t)(4 * DecodeTables<TYPE>::GC) * i));
  return v;
}
// Signs of eight values, two ways.  Both multiply where they could shift: the integer pipe that shifts, masks and permutes is
// what bounds these decoders, the one that multiplies has room.  `negate` takes the word whose bits 15 and 31 are those of pair P.
__device__ __forceinline__ uint32_t negate(uint32_t pair, uint32_t bits) { return pair ^ (bits & 0x80008000u); }
// ... from the sign bits themselves, s < 256: bit 2P to bit 15, bit 2P + 1 to bit 31 (the two products do not overlap)
template <int P> __device__ __forceinline__ uint32_t sign_bits8(uint32_t s) { return s * ((1u << (15 - 2 * P)) + (1u << (30 - 2 * P))); }
// ... from the table word of a 7-bit index: bits 15 - P and 31 - P
template <int TYPE> __device__ __forceinline__ uint32_t sign_word(const DecodeCtx& cx, uint32_t i) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(cx.sgn + (uint32_t)(4 * DecodeTables<TYPE>::SC) * i));
  return v;
}
template <int P> __device__ __forceinline__ uint32_t sign_bits(uint32_t word) { return word * (1u << P); }
__device__ __forceinline__ uint32_t iq_pair_signs(uint32_t sign_bits) {
  uint32_t w = 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) w |= ((sign_bits >> (2 * p)) & 1u) << (15 - p) | ((sign_bits >> (2 * p + 1)) & 1u) << (31 - p);
  return w;
}
// Shared-memory tables of the code-book decoders, built once per CTA from the formats' grid and sign tables.  An IQ2 grid entry
// holds eight magnitudes, each one of {8, 25, 43}; with the three products d*8, d*25, d*43 of a 32-value group rounded to 16 bits
// and parked in two registers, every PAIR of decoded values is one byte-permute whose selector depends only on the
// grid entry -- those selectors are what the table holds.
__device__ __forceinline__ uint4 iq2_pair_selectors(uint64_t grid_entry) {
  uint32_t s[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t m = (uint32_t)(grid_entry >> (8 * j)) & 0xFFu;
    const uint32_t c = (m > 8u ? 1u : 0u) + (m > 25u ? 1u : 0u);   // which of the three magnitudes
    const uint32_t nib = (2u * c) | ((2u * c + 1u) << 4);           // its two bytes in the register pair
    s[j >> 1] |= nib << (8 * (j & 1));
  }
  return make_uint4(s[0], s[1], s[2], s[3]);
}
// An IQ3 entry: its four magnitudes (at most 62) as 16-bit values, for fp16 divided by 256; those of IQ3_XXS are bf16 always (see Iq3Scale).
template <typename ab_t> __device__ __forceinline__ uint2 iq3_magnitudes(uint32_t g) {
  const float f = std::is_same<ab_t, __half>::value ? 1.f / 256.f : 1.f;
  return make_uint2(pack2<ab_t>(f * (float)(g & 0xFFu), f * (float)((g >> 8) & 0xFFu)), pack2<ab_t>(f * (float)((g >> 16) & 0xFFu), f * (float)(g >> 24)));
}

template <int TYPE, typename ab_t> __device__ __forceinline__ void decoder_fill_tables(uint8_t* tab) {
  using D = DecodeTables<TYPE>;
  if constexpr (D::GRID > 0) {
    for (int i = threadIdx.x; i < D::GRID * D::GC; i += blockDim.x) {
      const int e = i / D::GC;
      if constexpr (TYPE == T_IQ2_XXS) reinterpret_cast<uint4*>(tab)[i] = iq2_pair_selectors(d_iq2xxs_grid[e]);
      if constexpr (TYPE == T_IQ2_XS) reinterpret_cast<uint4*>(tab)[i] = iq2_pair_selectors(d_iq2xs_grid[e]);
      if constexpr (TYPE == T_IQ2_S) reinterpret_cast<uint4*>(tab)[i] = iq2_pair_selectors(d_iq2s_grid[e]);
      if constexpr (TYPE == T_IQ3_XXS) reinterpret_cast<uint2*>(tab)[i] = iq3_magnitudes<__nv_bfloat16>(d_iq3xxs_grid[e]);
      if constexpr (TYPE == T_IQ3_S) reinterpret_cast<uint2*>(tab)[i] = iq3_magnitudes<ab_t>(d_iq3s_grid[e]);
      if constexpr (TYPE == T_IQ1_S || TYPE == T_IQ1_M) reinterpret_cast<uint32_t*>(tab)[i] = d_iq1s_grid[e];
    }
  }
  if constexpr (D::SGN > 0) {
    uint32_t* sgn = reinterpret_cast<uint32_t*>(tab + D::GRID * D::GB * D::GC);
    for (int i = threadIdx.x; i < D::SGN * D::SC; i += blockDim.x) sgn[i] = iq_pair_signs(d_ksigns_iq2xs[i / D::SC]);
  }
}

template <int TYPE, typename ab_t> struct Decoder;
// formats decoded by the item (see Item128)
template <typename ab_t> struct Decoder<T_Q6_K, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ2_XXS, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ2_XS, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ2_S, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ3_XXS, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ3_S, ab_t> { static constexpr bool CORR = false; };
template <typename ab_t> struct Decoder<T_IQ4_NL, ab_t> { static constexpr bool CORR = false; };
template <> struct Decoder<T_IQ4_XS, __half> { static constexpr bool CORR = false; };
// types that are multiplied as dequantized weights of either 16-bit type (activations as they are)
template <int TYPE> __host__ __device__ constexpr bool decoder_bf16() {
  return TYPE == T_IQ2_XXS || TYPE == T_IQ2_XS || TYPE == T_IQ2_S || TYPE == T_IQ3_XXS || TYPE == T_IQ3_S || TYPE == T_IQ1_S || TYPE == T_IQ1_M ||
         TYPE == T_IQ4_NL || TYPE == T_IQ4_XS;
}

// Types whose two 32-value units of a 64-value stage (units 2j and 2j + 1 of a 256-value super-block, always
// whole) are cut from the same words of the block: load() depends on the unit only through u >> 1.
template <int TYPE> __host__ __device__ constexpr bool decoder_pair_load() { return TYPE == T_Q2_K || TYPE == T_Q3_K || TYPE == T_Q5_K; }

// one fp16 of each of four blocks TS bytes apart, zero from block `left` on
template <int TS> __device__ __forceinline__ uint2 block_halves(uint32_t a, int left) {
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = j < left ? lds16(a + TS * j) : 0u;
  return make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
}

// ---- Q4_0: value = half(q * d), q unsigned (see Stage64<T_Q4_0>); unit = one 18-byte block ----
template <typename ab_t> struct Decoder<T_Q4_0, ab_t> {
  static constexpr bool CORR = true;   // correction columns
  static constexpr int RW = 7;   // 18 bytes at 2-byte alignment: <= 6 words (+1 for the shifts)
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    ldg_cover<RW - 1>(row + (int64_t)u * 18, 18, raw);
    raw[RW - 1] = 0;
  }
  static __device__ __forceinline__ void decode(const uint8_t* row, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const uint32_t sh = shift_of(row + (int64_t)u * 18);
    const __half2 off = __floats2half2_rn(1024.f, 1024.f);
    const uint32_t du = word_at(raw, 0, sh) & 0xFFFFu;
    const __half2 d2 = u32_as_h2(du | (du << 16));
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // stream half-word 1+i holds qs[2i], qs[2i+1]
      const int h = 1 + i;
      const uint32_t wv = word_at(raw, h >> 1, sh);
      const uint32_t t = (h & 1) ? (wv >> 16) : (wv & 0xFFFFu);
      out[i] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024(t & 0xF, (t >> 8) & 0xF), off), d2));
      out[8 + i] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024((t >> 4) & 0xF, (t >> 12) & 0xF), off), d2));
    }
  }
  // d of the four blocks 4 * half .. of the chunk, of which `left` exist
  static __device__ __forceinline__ uint2 corr(const uint8_t* chunk, int half, int left) {
    return block_halves<18>(smem_u32(chunk) + 0 + 72 * half, left - 4 * half);
  }
};

// ---- Q8_0: value = half(q * d); unit = one 34-byte block ---------------------------------------
template <typename ab_t> struct Decoder<T_Q8_0, ab_t> {
  static constexpr bool CORR = false;   // correction columns
  static constexpr int RW = 11;  // 34 bytes: <= 10 words (+1)
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    ldg_cover<RW - 1>(row + (int64_t)u * 34, 34, raw);
    raw[RW - 1] = 0;
  }
  static __device__ __forceinline__ void decode(const uint8_t* row, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const uint32_t sh = shift_of(row + (int64_t)u * 34);
    const __half2 off = __floats2half2_rn(1152.f, 1152.f);  // 1024 + 128
    const uint32_t du = word_at(raw, 0, sh) & 0xFFFFu;
    const __half2 d2 = u32_as_h2(du | (du << 16));
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int h = 1 + i;
      const uint32_t wv = word_at(raw, h >> 1, sh);
      const uint32_t t = ((h & 1) ? (wv >> 16) : (wv & 0xFFFFu)) ^ 0x8080u;  // int8 -> biased unsigned
      out[i] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024(t & 0xFF, t >> 8), off), d2));
    }
  }
};

// 6-bit (scale, min) pair j of a Q4_K super-block from its 12 packed bytes held in three
// registers (bytes 0-3, 4-7, 8-11); same packing as get_scale_min_k4, dequantize.cuh:156-163.
__device__ __forceinline__ void q4k_scale_min(uint32_t w0, uint32_t w1, uint32_t w2, int j, int& sc, int& m) {
  if (j < 4) {
    sc = (w0 >> (8 * j)) & 63;
    m = (w1 >> (8 * j)) & 63;
  } else {
    const int sh = 8 * (j - 4);
    const uint32_t b = (w2 >> sh) & 0xFF;
    sc = (b & 0xF) | ((((w0 >> sh) & 0xFF) >> 6) << 4);
    m = (b >> 4) | ((((w1 >> sh) & 0xFF) >> 6) << 4);
  }
}

// half(dmin * m) of the sub-blocks 4 * half .. 4 * half + 3 of a Q4_K / Q5_K super-block with header h
__device__ __forceinline__ uint2 q4k_pair_mins(uint4 h, int half) {
  const uint32_t mn = half ? ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3F3F3F3Fu;   // four bytes
  const __half2 dmin = __half2half2(__ushort_as_half((unsigned short)(h.x >> 16))), off = __floats2half2_rn(1024.f, 1024.f);
  const __half2 a = __hsub2(u32_as_h2(__byte_perm(mn, 0x64646464u, 0x4140)), off), b = __hsub2(u32_as_h2(__byte_perm(mn, 0x64646464u, 0x4342)), off);
  return make_uint2(h2_as_u32(hmul2_rn(dmin, a)), h2_as_u32(hmul2_rn(dmin, b)));
}

// ---- Q4_K: A = half(d1 * q) with d1 = half(d * sc); the -dmin*m part is a correction column ----
// unit u: super-block u>>3, sub-block j = u&7: nibble (j&1) of the 32 bytes qs[32*(j>>1) ..]
template <typename ab_t> struct Decoder<T_Q4_K, ab_t> {
  static constexpr bool CORR = true;   // correction columns
  static constexpr int RW = 12;  // header (16 bytes) + 32 bytes of nibbles, all 16-byte aligned
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint8_t* blk = row + (int64_t)(u >> 3) * 144;
    const uint32_t sb = smem_u32(blk), sq = sb + 16 + 32 * ((u >> 1) & 3);
    const uint4 h = lds128s(sb), a = lds128s(sq), b = lds128s(sq + 16);
    raw[0] = h.x; raw[1] = h.y; raw[2] = h.z; raw[3] = h.w;
    raw[4] = a.x; raw[5] = a.y; raw[6] = a.z; raw[7] = a.w; raw[8] = b.x; raw[9] = b.y; raw[10] = b.z; raw[11] = b.w;
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const int j = u & 7, sh = 4 * (j & 1);
    const __half dall = __ushort_as_half((unsigned short)(raw[0] & 0xffff));
    int sc, m;
    q4k_scale_min(raw[1], raw[2], raw[3], j, sc, m);
    (void)m;
    const __half2 dv = __half2half2(__hmul_rn(dall, __int2half_rn(sc)));
    const __half2 off = __floats2half2_rn(1024.f, 1024.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // word i: bytes 4i..4i+3 -> values 4i..4i+3 of this sub-block
      const uint32_t w = raw[4 + i] >> sh;
      out[2 * i] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024(w & 0xF, (w >> 8) & 0xF), off), dv));
      out[2 * i + 1] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024((w >> 16) & 0xF, (w >> 24) & 0xF), off), dv));
    }
  }
  // half(dmin * m) of the four sub-blocks 4 * half .. of the chunk (pairs with -s8 on the B side)
  static __device__ __forceinline__ uint2 corr(const uint8_t* blk, int half, int) { return q4k_pair_mins(lds128s(smem_u32(blk)), half); }
};

// ---- Q4_1: A = half(q * d); the min term m * s8 is a correction column (B side: +s8) -----------------
template <typename ab_t> struct Decoder<T_Q4_1, ab_t> {
  static constexpr bool CORR = true;   // correction columns
  static constexpr int RW = 5;   // 20 bytes, 4-byte aligned
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint32_t sb = smem_u32(row + (int64_t)u * 20);
#pragma unroll
    for (int i = 0; i < 5; ++i) raw[i] = lds32(sb + 4u * i);
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const uint32_t du = raw[0] & 0xFFFFu;
    const __half2 d2 = u32_as_h2(du | (du << 16)), off = __floats2half2_rn(1024.f, 1024.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // word k = qs[4k..4k+3]: values 4k.. (low nibbles) and 16 + 4k.. (high); halves 1024 + code by byte-permute
      const uint32_t cl = raw[1 + k] & 0x0F0F0F0Fu, ch = (raw[1 + k] >> 4) & 0x0F0F0F0Fu;
      out[2 * k] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(cl, 0x64646464u, 0x4140)), off), d2));
      out[2 * k + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(cl, 0x64646464u, 0x4342)), off), d2));
      out[8 + 2 * k] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(ch, 0x64646464u, 0x4140)), off), d2));
      out[8 + 2 * k + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(ch, 0x64646464u, 0x4342)), off), d2));
    }
  }
  // m of the four blocks 4 * half .. of the chunk, of which `left` exist
  static __device__ __forceinline__ uint2 corr(const uint8_t* chunk, int half, int left) {
    return block_halves<20>(smem_u32(chunk) + 2 + 80 * half, left - 4 * half);
  }
};

// fifth bits: bit j of qh belongs to value j
// Word k of a 5-bit legacy block (qs[4k..4k+3]) -> the four pairs it holds: values 4k, 4k+1 | 4k+2, 4k+3 (low nibbles,
// fifth bits 4k.. of qh) and 16+4k.. (high nibbles, fifth bits 16+4k..).  Four consecutive bits of qh are spread to bit 4
// of four bytes with one multiplication (t * 0x02040810 puts bit j of t at bit 8j + 4, no carries for t < 16), the code
// bytes become halves 1024 + code by byte-permute, the offset is subtracted exactly and d multiplies once.
__device__ __forceinline__ void q5_word(uint32_t q, uint32_t qh, int k, __half2 off, __half2 d2, uint32_t& lo01, uint32_t& lo23,
                                        uint32_t& hi01, uint32_t& hi23) {
  const uint32_t cl = (q & 0x0F0F0F0Fu) | ((((qh >> (4 * k)) & 0xFu) * 0x02040810u) & 0x10101010u);
  const uint32_t ch = ((q >> 4) & 0x0F0F0F0Fu) | ((((qh >> (16 + 4 * k)) & 0xFu) * 0x02040810u) & 0x10101010u);
  lo01 = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(cl, 0x64646464u, 0x4140)), off), d2));
  lo23 = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(cl, 0x64646464u, 0x4342)), off), d2));
  hi01 = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(ch, 0x64646464u, 0x4140)), off), d2));
  hi23 = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(ch, 0x64646464u, 0x4342)), off), d2));
}

// ---- Q5_0: value = half((q - 16) * d), 22-byte blocks (2-byte aligned): d | qh[4] | qs[16] ------------
template <typename ab_t> struct Decoder<T_Q5_0, ab_t> {
  static constexpr bool CORR = false;   // correction columns
  static constexpr int RW = 8;   // 22 bytes at 2-byte alignment: <= 6 words (+ shifts)
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    ldg_cover<7>(row + (int64_t)u * 22, 22, raw);
    raw[7] = 0;
  }
  static __device__ __forceinline__ void decode(const uint8_t* row, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const uint32_t sh = shift_of(row + (int64_t)u * 22);
    const uint32_t w0 = word_at(raw, 0, sh), w1 = word_at(raw, 1, sh);
    const uint32_t du = w0 & 0xFFFFu, qh = (w0 >> 16) | (w1 << 16);
    const __half2 d2 = u32_as_h2(du | (du << 16)), off = __floats2half2_rn(1040.f, 1040.f);   // 1024 + 16
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // bytes 6 + 4k .. of the block = qs[4k..4k+3]: values 4k.. (low nibbles) and 16 + 4k.. (high)
      const uint32_t q = __funnelshift_r(word_at(raw, 1 + k, sh), word_at(raw, 2 + k, sh), 16);
      q5_word(q, qh, k, off, d2, out[2 * k], out[2 * k + 1], out[8 + 2 * k], out[8 + 2 * k + 1]);
    }
  }
};

// ---- Q5_1: A = half(q * d), 24-byte blocks (8-byte aligned): d | m | qh[4] | qs[16]; correction column m ----
template <typename ab_t> struct Decoder<T_Q5_1, ab_t> {
  static constexpr bool CORR = true;   // correction columns
  static constexpr int RW = 6;
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint32_t sb = smem_u32(row + (int64_t)u * 24);
    const uint2 a0 = lds64(sb), a1 = lds64(sb + 8), a2 = lds64(sb + 16);
    raw[0] = a0.x; raw[1] = a0.y; raw[2] = a1.x; raw[3] = a1.y; raw[4] = a2.x; raw[5] = a2.y;
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const uint32_t du = raw[0] & 0xFFFFu, qh = raw[1];
    const __half2 d2 = u32_as_h2(du | (du << 16)), off = __floats2half2_rn(1024.f, 1024.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) q5_word(raw[2 + k], qh, k, off, d2, out[2 * k], out[2 * k + 1], out[8 + 2 * k], out[8 + 2 * k + 1]);
  }
  // m of the four blocks 4 * half .. of the chunk, of which `left` exist
  static __device__ __forceinline__ uint2 corr(const uint8_t* chunk, int half, int left) {
    return block_halves<24>(smem_u32(chunk) + 2 + 96 * half, left - 4 * half);
  }
};

// ---- Q5_K: A = half(d1 * q), d1 = half(d * sc), q = 4 bits of qs | fifth bit of qh; -dmin*m is a correction column ----
// 176-byte blocks (16-byte aligned): d | dmin | scales[12] | qh[32] | qs[128].  unit u: sub-block j = u&7:
// nibble (j&1) of qs[32*(j>>1) + l], bit j of qh[l], l = 0..31.
template <typename ab_t> struct Decoder<T_Q5_K, ab_t> {
  static constexpr bool CORR = true;   // correction columns
  static constexpr int RW = 20;  // header (16) + 32 bytes of nibbles + 32 bytes of high bits
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint8_t* blk = row + (int64_t)(u >> 3) * 176;
    const uint32_t sb = smem_u32(blk), sq = sb + 48 + 32 * ((u >> 1) & 3);
    const uint4 h = lds128s(sb), a = lds128s(sq), b = lds128s(sq + 16), c = lds128s(sb + 16), e = lds128s(sb + 32);
    raw[0] = h.x; raw[1] = h.y; raw[2] = h.z; raw[3] = h.w;
    raw[4] = a.x; raw[5] = a.y; raw[6] = a.z; raw[7] = a.w; raw[8] = b.x; raw[9] = b.y; raw[10] = b.z; raw[11] = b.w;
    raw[12] = c.x; raw[13] = c.y; raw[14] = c.z; raw[15] = c.w; raw[16] = e.x; raw[17] = e.y; raw[18] = e.z; raw[19] = e.w;
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const int j = u & 7, sh = 4 * (j & 1);
    const __half dall = __ushort_as_half((unsigned short)(raw[0] & 0xffff));
    int sc, m;
    q4k_scale_min(raw[1], raw[2], raw[3], j, sc, m);
    (void)m;
    const __half2 dv = __half2half2(__hmul_rn(dall, __int2half_rn(sc)));
    const __half2 off = __floats2half2_rn(1024.f, 1024.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // word i: bytes 4i..4i+3 -> values 4i..4i+3 of this sub-block
      const uint32_t w = raw[4 + i] >> sh, hb = (raw[12 + i] >> j) & 0x01010101u;
      const uint32_t c0 = (w & 0xF) | ((hb & 1u) << 4), c1 = ((w >> 8) & 0xF) | (((hb >> 8) & 1u) << 4);
      const uint32_t c2 = ((w >> 16) & 0xF) | (((hb >> 16) & 1u) << 4), c3 = ((w >> 24) & 0xF) | (((hb >> 24) & 1u) << 4);
      out[2 * i] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024(c0, c1), off), dv));
      out[2 * i + 1] = h2_as_u32(hmul2_rn(__hsub2(ints_plus_1024(c2, c3), off), dv));
    }
  }
  // half(dmin * m) of the four sub-blocks 4 * half .. of the chunk (pairs with -s8 on the B side)
  static __device__ __forceinline__ uint2 corr(const uint8_t* blk, int half, int) { return q4k_pair_mins(lds128s(smem_u32(blk)), half); }
};

// ---- Q2_K: value = fp32 (d*sc)*q - dmin*m rounded once (the dequantized weight itself: the 16-value
// sub-blocks are finer than the 32-value sums of q8_1, so the min term cannot ride in a correction
// column); unit = 32-value group g = u&7 = 4n + j: bytes qs[32n..32n+31] >> 2j, scales 2g, 2g+1.
// A sub-block has only four possible values; they are rounded once each, parked in two registers
// as four halves, and every pair of weights is one byte-permute whose selector is the pair's two
// 2-bit codes times 0x22 plus 0x1010 (code c picks bytes 2c, 2c+1).
template <typename ab_t> struct Decoder<T_Q2_K, ab_t> {
  static constexpr bool CORR = false;   // correction columns
  static constexpr int RW = 10;   // 32 code bytes, the word holding the two scale bytes, (d, dmin): all 4-byte aligned
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint32_t sb = smem_u32(row + (int64_t)(u >> 3) * 84);
    const int g = u & 7;
    const uint32_t sq = sb + 16 + 32 * (g >> 2);
#pragma unroll
    for (int i = 0; i < 8; ++i) raw[i] = lds32(sq + 4u * i);
    raw[8] = lds32(sb + ((2 * g) & ~3));
    raw[9] = lds32(sb + 80);
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const int g = u & 7, sh = 2 * (g & 3);
    const float d = __half2float(__ushort_as_half((unsigned short)(raw[9] & 0xFFFFu)));
    const float dmin = __half2float(__ushort_as_half((unsigned short)(raw[9] >> 16)));
    const uint32_t sc2 = raw[8] >> (16 * (g & 1));
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {   // the two 16-value sub-blocks of the unit
      const uint32_t sc = (sc2 >> (8 * hb)) & 0xFFu;
      const float dl = d * (float)(sc & 0xFu), ml = dmin * (float)(sc >> 4);
      const uint32_t r0 = pack2<ab_t>(-ml, dl - ml), r1 = pack2<ab_t>(fmaf(2.f, dl, -ml), fmaf(3.f, dl, -ml));
#pragma unroll
      for (int i = 0; i < 4; ++i) {    // word 4hb + i: values 16hb + 4i .. + 3
        const uint32_t x = (raw[4 * hb + i] >> sh) & 0x03030303u;
        out[8 * hb + 2 * i] = __byte_perm(r0, r1, x * 0x22u + 0x1010u);
        out[8 * hb + 2 * i + 1] = __byte_perm(r0, r1, (x >> 16) * 0x22u + 0x1010u);
      }
    }
  }
};

// ---- Q3_K: value = d * ((sc6 - 32) * (c - 4)), c = 2 low bits | hmask bit << 2; unit = 32-value group
// g = u&7 = 4n + j: bytes qs[32n..32n+31] >> 2j, bit g of hmask[0..31], scales 2g, 2g+1.  Blocks are
// 110 bytes, so everything is read as covering words and realigned.  The code lands at bits 3-5 of
// a byte (two rotates, two masks per four weights), one byte-permute per pair turns it into the
// half 128 + c (0x5800 | c << 3), one HFMA2 gives (c - 4) * sc exactly (|.| <= 128; the addend
// -132 * sc has 11 significant bits) and the multiplication by d rounds once.
template <typename ab_t> struct Decoder<T_Q3_K, ab_t> {
  static constexpr bool CORR = false;   // correction columns
  static constexpr int RW = 26;   // [0..9] code words, [10..19] hmask words, [20..24] the 12 scale bytes, [25] d
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint8_t* blk = row + (int64_t)(u >> 3) * 110;
    const int g = u & 7;
    ldg_cover<9>(blk + 32 + 32 * (g >> 2), 32, raw);
    raw[9] = 0;
    ldg_cover<9>(blk, 32, raw + 10);
    raw[19] = 0;
    ldg_cover<4>(blk + 96, 12, raw + 20);
    raw[24] = 0;
    ldg_cover<1>(blk + 108, 2, raw + 25);
  }
  static __device__ __forceinline__ void decode(const uint8_t* row, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    static_assert(sizeof(ab_t) == 2 && std::is_same<ab_t, __half>::value, "Q3_K is decoded with fp16 arithmetic");
    const uint8_t* blk = row + (int64_t)(u >> 3) * 110;
    const int g = u & 7, k = g >> 1;
    const uint32_t sh_q = shift_of(blk + 32 + 32 * (g >> 2)), sh_h = shift_of(blk), sh_s = shift_of(blk + 96);
    // 6-bit scales 2g, 2g+1: low nibbles from byte 2g (mod 8) of the first eight scale bytes, shifted by
    // four for g >= 4; the two high bits from byte 2g mod 4 of the last four, bit pair g / 2
    const uint32_t a01 = word_at(raw + 20, k & 1, sh_s), tmp = word_at(raw + 20, 2, sh_s);
    const uint32_t us4 = ((a01 >> (4 * (k >> 1))) & 0x0F0F0F0Fu) | (((tmp >> (2 * k)) & 0x03030303u) << 4);
    const uint32_t us2 = us4 >> (16 * (g & 1));
    const uint32_t du = (raw[25] >> shift_of(blk + 108)) & 0xFFFFu;
    const __half2 d2 = u32_as_h2(du | (du << 16));
    const uint32_t rot_q = (uint32_t)(2 * (g & 3) - 3) & 31u, rot_h = (uint32_t)(g - 5) & 31u;
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
      const __half s = __int2half_rn((int)((us2 >> (8 * hb)) & 0xFFu) - 32);
      const __half2 s2 = __half2half2(s), c2 = __half2half2(__hmul(s, __float2half_rn(-132.f)));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t wq = word_at(raw, 4 * hb + i, sh_q), wh = word_at(raw + 10, 4 * hb + i, sh_h);
        const uint32_t c = (__funnelshift_r(wq, wq, rot_q) & 0x18181818u) | (__funnelshift_r(wh, wh, rot_h) & 0x20202020u);
        const __half2 p0 = u32_as_h2(__byte_perm(c, 0x58585858u, 0x4140)), p1 = u32_as_h2(__byte_perm(c, 0x58585858u, 0x4342));
        out[8 * hb + 2 * i] = h2_as_u32(hmul2_rn(__hfma2(p0, s2, c2), d2));
        out[8 * hb + 2 * i + 1] = h2_as_u32(hmul2_rn(__hfma2(p1, s2, c2), d2));
      }
    }
  }
};

// byte k of w (unsigned) as the float 2^23 + byte, without a conversion instruction
__device__ __forceinline__ float byte_2p23(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | k)); }
// The sixteen IQ4 levels plus 128 in four registers: two byte-permutes look four indices up in a half of the table each (the
// nibbles of q3, bit 3 cleared, are the selectors), a third takes the half that each index's top bit names.  Four bytes, in the
// order of the nibbles.
__device__ __forceinline__ uint32_t iq4_levels4(uint32_t q3, uint32_t sel) {
  return __byte_perm(__byte_perm(0x3F2D1801u, 0x766A5D4Fu, q3), __byte_perm(0xA6998D81u, 0xF1D9C5B5u, q3), sel);
}
// A word of IQ4 indices (values 4i.. in the low nibbles, 16 + 4i.. in the high ones) -> the two pairs of each, scaled in fp32 and rounded once
template <typename ab_t> __device__ __forceinline__ void iq4_word(uint32_t w, float dl, uint32_t* lo, uint32_t* hi) {
  const uint32_t q3 = w & 0x77777777u, sel = ((w & 0x88888888u) >> 1) | 0x32103210u;
  const uint32_t a = iq4_levels4(q3, sel), b = iq4_levels4(q3 >> 16, sel >> 16);   // bytes (4i, 16+4i, 4i+1, 17+4i) and (4i+2, ...)
  auto v = [&](uint32_t x, int k) { return dl * (byte_2p23(x, k) - 8388736.f); };   // 2^23 + 128
  lo[0] = pack2<ab_t>(v(a, 0), v(a, 2));
  lo[1] = pack2<ab_t>(v(b, 0), v(b, 2));
  hi[0] = pack2<ab_t>(v(a, 1), v(a, 3));
  hi[1] = pack2<ab_t>(v(b, 1), v(b, 3));
}

// ---- IQ4_XS with bf16 activations: fp32 d*(ls-32)*level rounded once; unit = 32-value group ib = u&7 -----------
template <> struct Decoder<T_IQ4_XS, __nv_bfloat16> {
  static constexpr bool CORR = false;
  static constexpr int RW = 6;   // header (8 bytes) + 16 index bytes, 8-byte aligned
  static __device__ __forceinline__ void load(const uint8_t* row, int u, uint32_t (&raw)[RW]) {
    const uint8_t* blk = row + (int64_t)(u >> 3) * 136;
    const uint32_t sb = smem_u32(blk);
    const uint2 h = lds64(sb), a = lds64(sb + 8 + 16 * (u & 7)), b = lds64(sb + 16 + 16 * (u & 7));
    raw[0] = h.x; raw[1] = h.y; raw[2] = a.x; raw[3] = a.y; raw[4] = b.x; raw[5] = b.y;
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int u, const uint32_t (&raw)[RW], const DecodeCtx&, uint32_t (&out)[16]) {
    const int ib = u & 7;
    const float d = __half2float(__ushort_as_half((unsigned short)(raw[0] & 0xffff)));
    const int ls = (int)(((raw[1] >> (4 * ib)) & 0xF) | ((((raw[0] >> 16) >> (2 * ib)) & 3) << 4)) - 32;
    const float dl = d * (float)ls;
#pragma unroll
    for (int i = 0; i < 4; ++i) iq4_word<__nv_bfloat16>(raw[2 + i], dl, out + 2 * i, out + 8 + 2 * i);
  }
};

// 8 values of an IQ1 entry (codes 0, 1, 2 in nibbles: values 0-3 low, 4-7 high): the group has three possible values d * (code +
// delta), rounded once each and parked in r0, r1; a pair is one byte-permute whose selector is its codes times 0x22 plus 0x1010
__device__ __forceinline__ void iq1_entry(uint32_t g, uint32_t r0, uint32_t r1, uint32_t* out) {
  const uint32_t s0 = (g & 0x0F0F0F0Fu) * 0x22u + 0x10101010u, s1 = ((g >> 4) & 0x0F0F0F0Fu) * 0x22u + 0x10101010u;
  out[0] = __byte_perm(r0, r1, s0);
  out[1] = __byte_perm(r0, r1, s0 >> 16);
  out[2] = __byte_perm(r0, r1, s1);
  out[3] = __byte_perm(r0, r1, s1 >> 16);
}
template <typename ab_t> struct Decoder<T_IQ1_S, ab_t> {   // half d | u8 qs[32] | u16 qh[8], 50 bytes
  static constexpr bool CORR = false;
  static constexpr int RW = 4;
  static __device__ __forceinline__ void load(const uint8_t* blk, int u, uint32_t (&raw)[RW]) {
    ldg_cover<1>(blk, 2, raw);
    ldg_cover<2>(blk + 2 + 4 * u, 4, raw + 1);
    ldg_cover<1>(blk + 34 + 2 * u, 2, raw + 3);
  }
  static __device__ __forceinline__ void decode(const uint8_t* blk, int u, const uint32_t (&raw)[RW], const DecodeCtx& cx, uint32_t (&out)[16]) {
    const float dh = __half2float(__ushort_as_half((unsigned short)((raw[0] >> shift_of(blk)) & 0xFFFFu)));
    const uint32_t q = word_at(raw + 1, 0, shift_of(blk + 2 + 4 * u)), qh = (raw[3] >> shift_of(blk + 34 + 2 * u)) & 0xFFFFu;
    const float d = dh * (float)(2u * ((qh >> 12) & 7u) + 1u), delta = qh & 0x8000u ? -1.125f : -0.875f;
    const uint32_t r0 = pack2<ab_t>(d * delta, d * (1.f + delta)), r1 = pack2<ab_t>(d * (2.f + delta), 0.f);
#pragma unroll
    for (int l = 0; l < 4; ++l) iq1_entry(grid32<T_IQ1_S>(cx, ((q >> (8 * l)) & 0xFFu) | (((qh >> (3 * l)) & 7u) << 8)), r0, r1, out + 4 * l);
  }
};
template <typename ab_t> struct Decoder<T_IQ1_M, ab_t> {   // u8 qs[32] | u8 qh[16] | u16 scales[4], 56 bytes (8-byte aligned)
  static constexpr bool CORR = false;
  static constexpr int RW = 4;
  static __device__ __forceinline__ void load(const uint8_t* blk, int u, uint32_t (&raw)[RW]) {
    const uint32_t sb = smem_u32(blk);
    raw[0] = lds32(sb + 4 * u);
    raw[1] = (lds32(sb + 32 + 4 * (u >> 1)) >> (16 * (u & 1))) & 0xFFFFu;
    const uint2 s = lds64(sb + 48);
    raw[2] = s.x; raw[3] = s.y;
  }
  static __device__ __forceinline__ void decode(const uint8_t*, int u, const uint32_t (&raw)[RW], const DecodeCtx& cx, uint32_t (&out)[16]) {
    const uint32_t s16 = ((raw[2] >> 12) & 0x000Fu) | ((raw[2] >> 24) & 0x00F0u) | ((raw[3] >> 4) & 0x0F00u) | ((raw[3] >> 16) & 0xF000u);
    const float dh = __half2float(__ushort_as_half((unsigned short)s16));
    const uint32_t s2 = ((u & 4) ? raw[3] : raw[2]) >> (16 * ((u >> 1) & 1) + 6 * (u & 1));
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t h = raw[1] >> (4 * l);
      const float d = dh * (float)(2u * ((s2 >> (3 * (l >> 1))) & 7u) + 1u), delta = h & 8u ? -1.125f : -0.875f;
      iq1_entry(grid32<T_IQ1_M>(cx, ((raw[0] >> (8 * l)) & 0xFFu) | ((h & 7u) << 8)), pack2<ab_t>(d * delta, d * (1.f + delta)),
                pack2<ab_t>(d * (2.f + delta), 0.f), out + 4 * l);
    }
  }
};

// =============================================================================================
// Whole-stage decoders: one thread turns the 64 values of one weight row of one K stage into
// the 128 bytes of that row in the A tile (out[4c..4c+3] = 16-byte piece c of the row).
//
// The specialised ("fast") forms read a dense 256-value chunk of the row from shared memory
// (the 2-D TMA box of mmq.cu) with 16-byte loads at compile-time offsets and build fp16 pairs
// with the mantissa trick: OR-ing a small unsigned integer n into the mantissa of 1024.0
// (0x6400) gives exactly 1024 + n, into bits 4-7 of 64.0 (0x5400) exactly 64 + n.  Values are
// the same as the 32-value decoders above produce (one rounding, in the final multiply).
//
// PERM: order of the 64 values inside the stage.  0 = natural.  1 = within every group of four
// consecutive values the middle two are swapped (0,2,1,3): the two low nibbles that sit 16 bits
// apart in a 32-bit word of packed bytes become one fp16 pair with a single AND/OR.  The
// activation matrix is written in the same order (quantize_q8_1.cu), so the contraction is
// unchanged.
// =============================================================================================
// Where the stage's number only moves addresses and shifts it is a run-time argument (one copy of the code for all four groups: the
// kernel's first pass over its instructions costs more than a stage); where it moves words between registers it is a template
// argument of stage<SC>().
template <int TYPE, typename ab_t> struct Stage64 {
  static constexpr bool FAST = false;
  static constexpr int PERM = 0;
};

__device__ __forceinline__ uint4 lds128(const uint8_t* p) { return lds128s(smem_u32(p)); }
__device__ __forceinline__ __half2 h2const(float v) { return __floats2half2_rn(v, v); }

// ---- Q4_K: chunk = one 144-byte super-block; stage SC = sub-blocks 2SC (low nibbles) and 2SC+1 ----
// the scales of the sub-blocks 2 * sc and 2 * sc + 1 of a Q4_K / Q5_K super-block, times d
__device__ __forceinline__ void q4k_pair_scales(uint4 h, int sc, __half& d0, __half& d1) {
  const __half dall = __ushort_as_half((unsigned short)(h.x & 0xffff));
  const int sh = 16 * (sc & 1);
  const uint32_t a = h.y >> sh, c = h.w >> sh;
  const uint32_t s2 = sc < 2 ? a & 0x3F3Fu : (c & 0x0F0Fu) | ((a >> 2) & 0x3030u);
  d0 = __hmul_rn(dall, __int2half_rn((int)(s2 & 0xFFu)));
  d1 = __hmul_rn(dall, __int2half_rn((int)(s2 >> 8)));
}
template <> struct Stage64<T_Q4_K, __half> {
  static constexpr bool FAST = true;
  static constexpr int PERM = 1;
  static __device__ __forceinline__ void decode(const uint8_t* blk, int sc, uint32_t (&out)[32]) {
    const uint4 h = lds128(blk);
    const uint4 qa = lds128(blk + 16 + 32 * sc), qb = lds128(blk + 32 + 32 * sc);
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
    __half d0, d1;
    q4k_pair_scales(h, sc, d0, d1);
    const __half2 s0 = __half2half2(d0), s1 = __half2half2(d1);
    const float big = fmaxf(fabsf(__half2float(d0)), fabsf(__half2float(d1)));
    if (big < 32.f) {
      // (1024 + n) * s - 1024 * s: the product term is exact, so this is n * s rounded once
      const __half2 c0 = __hmul2_rn(s0, h2const(-1024.f)), c1 = __hmul2_rn(s1, h2const(-64.f));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = w[j], b = w[j] >> 8;
        out[2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x000F000Fu) | 0x64006400u), s0, c0));
        out[2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x000F000Fu) | 0x64006400u), s0, c0));
        out[16 + 2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x00F000F0u) | 0x54005400u), s1, c1));
        out[16 + 2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x00F000F0u) | 0x54005400u), s1, c1));
      }
    } else {  // 1024 * s would overflow fp16: subtract the offset first (exact), then scale
      const __half2 o0 = h2const(1024.f), o1 = h2const(64.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = w[j], b = w[j] >> 8;
        out[2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x000F000Fu) | 0x64006400u), o0), s0));
        out[2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x000F000Fu) | 0x64006400u), o0), s0));
        out[16 + 2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x00F000F0u) | 0x54005400u), o1), s1));
        out[16 + 2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x00F000F0u) | 0x54005400u), o1), s1));
      }
    }
  }
};

// ---- Q5_K: chunk = one 176-byte super-block (d, dmin, 12 scale bytes, 32 bytes of fifth bits, 128 bytes of
// nibbles); stage SC = sub-blocks 2SC (low nibbles of qs[32SC..], bit 2SC of qh[l]) and 2SC+1 (high nibbles,
// bit 2SC+1).  As Q4_K with one more AND/OR per pair: the fifth bit lands at mantissa bit 4 of 1024 + n
// (low nibbles) or at mantissa bit 8 of 64 + n / 16 (high nibbles, n sits four bits up).
template <> struct Stage64<T_Q5_K, __half> {
  static constexpr bool FAST = true;
  static constexpr int PERM = 1;
  static __device__ __forceinline__ void decode(const uint8_t* blk, int sc, uint32_t (&out)[32]) {
    const uint4 h = lds128(blk);
    const uint4 ha = lds128(blk + 16), hb = lds128(blk + 32);
    const uint4 qa = lds128(blk + 48 + 32 * sc), qb = lds128(blk + 64 + 32 * sc);
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
    const uint32_t hw[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
    __half d0, d1;
    q4k_pair_scales(h, sc, d0, d1);
    const __half2 s0 = __half2half2(d0), s1 = __half2half2(d1);
    const float big = fmaxf(fabsf(__half2float(d0)), fabsf(__half2float(d1)));
    if (big < 32.f) {
      // (1024 + n) * s - 1024 * s: the product term is exact, so this is n * s rounded once
      const __half2 c0 = __hmul2_rn(s0, h2const(-1024.f)), c1 = __hmul2_rn(s1, h2const(-64.f));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = w[j], b = w[j] >> 8;
        const uint32_t x = hw[j] >> (2 * sc), y = hw[j] >> (2 * sc + 8);   // fifth bits of values (4j, 4j+2) / (4j+1, 4j+3) at bits 0 and 16
        out[2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x000F000Fu) | ((x << 4) & 0x00100010u) | 0x64006400u), s0, c0));
        out[2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x000F000Fu) | ((y << 4) & 0x00100010u) | 0x64006400u), s0, c0));
        out[16 + 2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x00F000F0u) | ((x << 7) & 0x01000100u) | 0x54005400u), s1, c1));
        out[16 + 2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x00F000F0u) | ((y << 7) & 0x01000100u) | 0x54005400u), s1, c1));
      }
    } else {  // 1024 * s would overflow fp16: subtract the offset first (exact), then scale
      const __half2 o0 = h2const(1024.f), o1 = h2const(64.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = w[j], b = w[j] >> 8;
        const uint32_t x = hw[j] >> (2 * sc), y = hw[j] >> (2 * sc + 8);
        out[2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x000F000Fu) | ((x << 4) & 0x00100010u) | 0x64006400u), o0), s0));
        out[2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x000F000Fu) | ((y << 4) & 0x00100010u) | 0x64006400u), o0), s0));
        out[16 + 2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x00F000F0u) | ((x << 7) & 0x01000100u) | 0x54005400u), o1), s1));
        out[16 + 2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x00F000F0u) | ((y << 7) & 0x01000100u) | 0x54005400u), o1), s1));
      }
    }
  }
};

// ---- Q4_0: chunk = 8 blocks of 18 bytes; stage SC = blocks 2SC, 2SC+1 at byte 36*SC ----------------
template <> struct Stage64<T_Q4_0, __half> {
  static constexpr bool FAST = true;
  static constexpr int PERM = 1;
  // The operand is half(q * d) with the UNSIGNED code q = 0..15 (the "- 8" of the format rides in the
  // correction column: -8 * d * s8, which is the reference's own tiled formula d * (sumi * d8 - 8 * s8),
  // vecdotq.cuh:61-64), so one HFMA2 makes a pair: (1024 + q) * d - 1024 * d is q * d rounded once.
  static __device__ __forceinline__ void block(const uint32_t (&q)[4], __half2 d2, uint32_t* out) {
    const float ad = fabsf(__low2float(d2));
    if (ad < 32.f) {
      const __half2 c0 = __hmul2_rn(d2, h2const(-1024.f)), c1 = __hmul2_rn(d2, h2const(-64.f));   // exact
#pragma unroll
      for (int j = 0; j < 4; ++j) {   // bytes 4j..4j+3: low nibbles = values 4j.., high nibbles = values 16+4j..
        const uint32_t a = q[j], b = q[j] >> 8;
        out[2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x000F000Fu) | 0x64006400u), d2, c0));
        out[2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x000F000Fu) | 0x64006400u), d2, c0));
        out[8 + 2 * j] = h2_as_u32(__hfma2(u32_as_h2((a & 0x00F000F0u) | 0x54005400u), d2, c1));
        out[8 + 2 * j + 1] = h2_as_u32(__hfma2(u32_as_h2((b & 0x00F000F0u) | 0x54005400u), d2, c1));
      }
    } else {   // 1024 * d would overflow fp16: subtract the offset first (exact), then scale
      const __half2 o0 = h2const(1024.f), o1 = h2const(64.f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t a = q[j], b = q[j] >> 8;
        out[2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x000F000Fu) | 0x64006400u), o0), d2));
        out[2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x000F000Fu) | 0x64006400u), o0), d2));
        out[8 + 2 * j] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((a & 0x00F000F0u) | 0x54005400u), o1), d2));
        out[8 + 2 * j + 1] = h2_as_u32(hmul2_rn(__hsub2(u32_as_h2((b & 0x00F000F0u) | 0x54005400u), o1), d2));
      }
    }
  }
  template <int SC> static __device__ __forceinline__ void stage(const uint8_t* chunk, uint32_t (&out)[32]) {
    constexpr int A0 = (36 * SC) & ~15, O = (36 * SC - A0) / 4;   // aligned start, word offset of block 2SC
    uint32_t W[12];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint4 v = lds128(chunk + A0 + 16 * i);
      W[4 * i] = v.x; W[4 * i + 1] = v.y; W[4 * i + 2] = v.z; W[4 * i + 3] = v.w;
    }
    // block 2SC starts at word O (d in the low half, nibbles 2 bytes in); block 2SC+1 at word O+4, upper half
    const uint32_t da = W[O] & 0xFFFFu, db = W[O + 4] >> 16;
    const uint32_t qa[4] = {__funnelshift_r(W[O], W[O + 1], 16), __funnelshift_r(W[O + 1], W[O + 2], 16),
                            __funnelshift_r(W[O + 2], W[O + 3], 16), __funnelshift_r(W[O + 3], W[O + 4], 16)};
    const uint32_t qb[4] = {W[O + 5], W[O + 6], W[O + 7], W[O + 8]};
    block(qa, u32_as_h2(da | (da << 16)), out);
    block(qb, u32_as_h2(db | (db << 16)), out + 16);
  }
  static __device__ __forceinline__ void decode(const uint8_t* chunk, int sc, uint32_t (&out)[32]) {
    switch (sc) {
      case 0: stage<0>(chunk, out); break;
      case 1: stage<1>(chunk, out); break;
      case 2: stage<2>(chunk, out); break;
      default: stage<3>(chunk, out); break;
    }
  }
};

// ---- Q8_0: chunk = 8 blocks of 34 bytes; stage SC = blocks 2SC, 2SC+1 at byte 68*SC ----------------
template <> struct Stage64<T_Q8_0, __half> {
  static constexpr bool FAST = true;
  static constexpr int PERM = 0;
  // two int8 codes (already biased by +128) -> (1024 + u0, 1024 + u1) -> (u - 128) * d
  static __device__ __forceinline__ uint32_t pair(uint32_t w, uint32_t sel, __half2 d2) {
    const __half2 o = h2const(1152.f);
    return h2_as_u32(hmul2_rn(__hsub2(u32_as_h2(__byte_perm(w, 0x64646464u, sel)), o), d2));
  }
  template <int SC> static __device__ __forceinline__ void stage(const uint8_t* chunk, uint32_t (&out)[32]) {
    constexpr int A0 = (68 * SC) & ~15, O = (68 * SC - A0) / 4;
    uint32_t W[20];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const uint4 v = lds128(chunk + A0 + 16 * i);
      W[4 * i] = v.x; W[4 * i + 1] = v.y; W[4 * i + 2] = v.z; W[4 * i + 3] = v.w;
    }
    const uint32_t da = W[O] & 0xFFFFu, db = W[O + 8] >> 16;
    const __half2 d2a = u32_as_h2(da | (da << 16)), d2b = u32_as_h2(db | (db << 16));
    // block 2SC: codes start in the upper half of word O; pair t = codes 2t, 2t+1 = half-word 1+t of the block
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const uint32_t wv = W[O + ((1 + t) >> 1)] ^ 0x80808080u;
      out[t] = pair(wv, ((1 + t) & 1) ? 0x4342u : 0x4140u, d2a);
    }
    // block 2SC+1: codes start at word O+9, aligned
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      const uint32_t wv = W[O + 9 + (t >> 1)] ^ 0x80808080u;
      out[16 + t] = pair(wv, (t & 1) ? 0x4342u : 0x4140u, d2b);
    }
  }
  static __device__ __forceinline__ void decode(const uint8_t* chunk, int sc, uint32_t (&out)[32]) {
    switch (sc) {
      case 0: stage<0>(chunk, out); break;
      case 1: stage<1>(chunk, out); break;
      case 2: stage<2>(chunk, out); break;
      default: stage<3>(chunk, out); break;
    }
  }
};

// =============================================================================================
// Item decoders: one thread turns half a 256-value chunk of its row, two stages, into operand A, whatever the row's alignment.
// What both stages need is read once (begin), and the 32-value units are dealt to the stages as suits the format: the
// activation matrix is written in that order (PERM, see mmq_perm).
//
// The N words of a row from the 2-byte aligned shared address a.  wide: every row of the tile has the same remainder modulo 16
// (rows that are a multiple of 16 bytes, as with most K): the slots are an odd number of 16-byte units apart, so 32-bit loads of
// 32 rows meet in eight banks, four at a time, and 16-byte loads do not.
// =============================================================================================
template <int N> __device__ __forceinline__ void lds_row_words(uint32_t a, bool wide, uint32_t (&w)[N]) {
  const uint32_t sh = (a & 2u) * 8u;
  if (wide) {
    constexpr int Q = (N + 7) / 4;
    uint32_t t[4 * Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const uint4 v = lds128s((a & ~15u) + 16u * i);
      t[4 * i] = v.x; t[4 * i + 1] = v.y; t[4 * i + 2] = v.z; t[4 * i + 3] = v.w;
    }
    switch ((a >> 2) & 3u) {
#define LDS_ROW_CASE(K) \
  _Pragma("unroll") for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(t[i + K], t[i + K + 1], sh); \
  break
      case 0: LDS_ROW_CASE(0);
      case 1: LDS_ROW_CASE(1);
      case 2: LDS_ROW_CASE(2);
      default: LDS_ROW_CASE(3);
#undef LDS_ROW_CASE
    }
  } else {
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) r[i] = lds32((a & ~3u) + 4u * i);
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(r[i], r[i + 1], sh);
  }
}

template <int TYPE, typename ab_t> struct Item128 { static constexpr bool HAVE = false; };

// ---- Q6_K: value = half(d * half(sc * (code - 32))), 210-byte blocks: ql[128] | qh[64] | sc[16] | d -----------------------
// Half ip has four units q of 32 values: low 4 bits = nibble q >> 1 of ql[64 ip + 32 (q & 1) + l], high 2 bits = bits 2q.. of
// qh[32 ip + l], scales sc[8 ip + 2q] (l < 16) and sc[8 ip + 2q + 1].  Stage h takes the units h and h + 2 -- both nibbles of the
// same 32 bytes -- so 16 words give 64 values (with units h and h + 1, all 64 bytes of ql were read twice).  The code goes to bits 2-7 of a byte;
// with 0x5C above it that is the half 256 + code, and (256 + code) * sc - 288 * sc is exact before its one rounding: 9 * 32 * sc has 11 significant bits.
template <typename ab_t> struct Item128<T_Q6_K, ab_t> {
  static constexpr bool HAVE = true;
  struct State {
    uint32_t h[8], sc[2];
    __half2 d2;
  };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<8>(row + 128 + 32 * ip, wide, s.h);
    lds_words_unaligned<2>(row + 192 + 8 * ip, s.sc);
    const uint32_t du = lds16(row + 208);
    s.d2 = u32_as_h2(du | (du << 16));
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t row, int ip, bool wide, const DecodeCtx&, const State& s, uint32_t (&out)[32]) {
    uint32_t l[8];
    lds_row_words<8>(row + 64 * ip + 32 * H, wide, l);
    __half2 sc[4], off[4];   // of the unit H, first and second 16 values, and of the unit H + 2
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sc[i] = __hsub2(u32_as_h2(__byte_perm(s.sc[i >> 1] ^ 0x80808080u, 0x64646464u, 0x4040u + 0x0101u * (2 * H + (i & 1)))), __floats2half2_rn(1152.f, 1152.f));
      off[i] = hmul2_rn(sc[i], __floats2half2_rn(-288.f, -288.f));
    }
#pragma unroll
    for (int w = 0; w < 8; ++w) {   // values 4w .. 4w + 3 of both units
      const uint32_t c0 = ((l[w] << 2) & 0x3C3C3C3Cu) | ((s.h[w] << (6 - 2 * H)) & 0xC0C0C0C0u);
      const uint32_t c1 = ((l[w] >> 2) & 0x3C3C3C3Cu) | ((s.h[w] << (2 - 2 * H)) & 0xC0C0C0C0u);
      const int i = w >> 2;
      out[2 * w] = h2_as_u32(hmul2_rn(s.d2, __hfma2(u32_as_h2(__byte_perm(c0, 0x5C5C5C5Cu, 0x4140)), sc[i], off[i])));
      out[2 * w + 1] = h2_as_u32(hmul2_rn(s.d2, __hfma2(u32_as_h2(__byte_perm(c0, 0x5C5C5C5Cu, 0x4342)), sc[i], off[i])));
      out[16 + 2 * w] = h2_as_u32(hmul2_rn(s.d2, __hfma2(u32_as_h2(__byte_perm(c1, 0x5C5C5C5Cu, 0x4140)), sc[2 + i], off[2 + i])));
      out[16 + 2 * w + 1] = h2_as_u32(hmul2_rn(s.d2, __hfma2(u32_as_h2(__byte_perm(c1, 0x5C5C5C5Cu, 0x4342)), sc[2 + i], off[2 + i])));
    }
  }
};

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return __byte_perm(w, 0u, 0x4440u | (uint32_t)k); }
// byte K of w with byte K of `high`, 0 or 1, above it, in one permute (a selector with bit 3 set replicates that byte's sign: zero)
template <int K> __device__ __forceinline__ uint32_t byte_of9(uint32_t w, uint32_t high) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(high), "n"(K | (4 + K) << 4 | (12 + K) << 8 | (12 + K) << 12));
  return r;
}
__device__ __forceinline__ uint32_t spread_bits4(uint32_t b) { return ((b & 0xFu) * 0x00204081u) & 0x01010101u; }   // bit j -> bit 0 of byte j

// ---- the IQ2 formats: value = +-round(d * magnitude), d = dh * (0.5 + s) * 0.25 in fp32, rounded once as in the reference (multiplying
// by -1.f afterwards is exact, so flipping the sign bit is the same) ----
template <typename ab_t> struct Iq2Group {   // the three possible magnitudes of a group, each rounded once
  uint32_t r0, r1;
  __device__ __forceinline__ void set(float dh, uint32_t s) {
    const float d = dh * (0.5f + (float)s) * 0.25f;
    r0 = pack2<ab_t>(d * 8.f, d * 25.f);
    r1 = pack2<ab_t>(d * 43.f, 0.f);
  }
};
template <typename ab_t> __device__ __forceinline__ void iq2_entry(const Iq2Group<ab_t>& g, uint4 sel, uint32_t word, uint32_t* out) {
  out[0] = negate(__byte_perm(g.r0, g.r1, sel.x), sign_bits<0>(word));
  out[1] = negate(__byte_perm(g.r0, g.r1, sel.y), sign_bits<1>(word));
  out[2] = negate(__byte_perm(g.r0, g.r1, sel.z), sign_bits<2>(word));
  out[3] = negate(__byte_perm(g.r0, g.r1, sel.w), sign_bits<3>(word));
}
template <typename ab_t> struct Item128<T_IQ2_XXS, ab_t> {   // half d | per 32 values: four grid bytes, four 7-bit sign indices and a 4-bit scale; 66 bytes
  static constexpr bool HAVE = true;
  struct State { uint32_t q[8]; float dh; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<8>(row + 2 + 32 * ip, wide, s.q);
    s.dh = lds_half_f32(row);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx& cx, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t idx = s.q[4 * H + 2 * u], aux = s.q[4 * H + 2 * u + 1];
      Iq2Group<ab_t> g;
      g.set(s.dh, aux >> 28);
#pragma unroll
      for (int l = 0; l < 4; ++l)
        iq2_entry<ab_t>(g, grid128<T_IQ2_XXS>(cx, byte_of(idx, l)), sign_word<T_IQ2_XXS>(cx, (aux >> (7 * l)) & 127u), out + 16 * u + 4 * l);
    }
  }
};
template <typename ab_t> struct Item128<T_IQ2_XS, ab_t> {   // half d | u16 qs[32] | u8 scales[8], 74 bytes
  static constexpr bool HAVE = true;
  struct State { uint32_t q[8], sc; float dh; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<8>(row + 2 + 32 * ip, wide, s.q);
    uint32_t w[1];
    lds_words_unaligned<1>(row + 66 + 4 * ip, w);
    s.sc = w[0];
    s.dh = lds_half_f32(row);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx& cx, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {   // 16 values: a word of indices, half a byte of scales
      const uint32_t q = s.q[4 * H + v];
      Iq2Group<ab_t> g;
      g.set(s.dh, (s.sc >> (16 * H + 4 * v)) & 0xFu);
#pragma unroll
      for (int l = 0; l < 2; ++l)
        iq2_entry<ab_t>(g, grid128<T_IQ2_XS>(cx, (q >> (16 * l)) & 511u), sign_word<T_IQ2_XS>(cx, (q >> (16 * l + 9)) & 127u), out + 8 * v + 4 * l);
    }
  }
};
template <typename ab_t> struct Item128<T_IQ2_S, ab_t> {   // half d | u8 qs[32] | u8 signs[32] | u8 qh[8] | u8 scales[8], 82 bytes
  static constexpr bool HAVE = true;
  struct State { uint32_t q[4], sg[4], qh, sc; float dh; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<4>(row + 2 + 16 * ip, wide, s.q);
    lds_row_words<4>(row + 34 + 16 * ip, wide, s.sg);
    uint32_t w[1];
    lds_words_unaligned<1>(row + 66 + 4 * ip, w);
    s.qh = w[0];
    lds_words_unaligned<1>(row + 74 + 4 * ip, w);
    s.sc = w[0];
    s.dh = lds_half_f32(row);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx& cx, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t q = s.q[2 * H + u], sg = s.sg[2 * H + u], qh = s.qh >> (16 * H + 8 * u);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Iq2Group<ab_t> g;
        g.set(s.dh, (s.sc >> (16 * H + 8 * u + 4 * h)) & 0xFu);
#pragma unroll
        for (int l2 = 0; l2 < 2; ++l2) {
          const int l = 2 * h + l2;
          const uint4 sel = grid128<T_IQ2_S>(cx, byte_of(q, l) | ((qh << (8 - 2 * l)) & 0x300u));
          const uint32_t sb = byte_of(sg, l);
          uint32_t* o = out + 16 * u + 4 * l;
          o[0] = negate(__byte_perm(g.r0, g.r1, sel.x), sign_bits8<0>(sb));
          o[1] = negate(__byte_perm(g.r0, g.r1, sel.y), sign_bits8<1>(sb));
          o[2] = negate(__byte_perm(g.r0, g.r1, sel.z), sign_bits8<2>(sb));
          o[3] = negate(__byte_perm(g.r0, g.r1, sel.w), sign_bits8<3>(sb));
        }
      }
    }
  }
};

// ---- the IQ3 formats: value = +-round(d * magnitude), d = dh * (0.5 + s) * 0.5 in fp32 (at most 16 significant bits) ----
// (8192x28672, 300 tokens, bf16, products split in bf16 at the time: 121.4 -> 112.5 us with the same plan; in fp32 as now the call keeps its gain, 149.9 -> 138.5 against 148.4 -> 137.1; 165 -> about 100 shared-memory wavefronts a stage of 32 rows; the
// IQ2 formats with their signs as above, IQ2_XXS 28672x8192, 128 tokens: 67.9 -> 61.8 us.)
// IQ3_S with fp16: two 16-bit instructions a pair instead of two permutes, two fp32 multiply-adds and a conversion.  d is the sum of two 16-bit
// numbers and fma(m, hi, m * lo) rounds the sum once: lo has at most five significant bits, m four, so m * lo is exact and the result the correctly
// rounded one.  The magnitudes are held divided by 256 and d times 256, which keeps lo clear of the subnormals; a d beyond that range takes the
// fp32 form (`wide`).
// bf16, and IQ3_XXS: the product in fp32, exact in 21 bits, two values an instruction, rounded once; the magnitudes are held in bf16 (five bits).
// Split in bf16, m * lo would be rounded to eight bits before the sum (0.502 of a last place against 0.500, one weight in 2500); of IQ3_XXS in fp16 62 / 256 * lo can be
// an odd multiple of 2^-25, half of fp16's last place, where dh is below 2^-13, and taking the fp32 form only there made warps run both
// (14336x4096, 512 tokens: 70.7 us against 63.1 before all this).
// Iq3Scale: magnitudes in MT times d in fp32, as ab_t
template <typename MT, typename ab_t> struct Iq3Scale {
  uint64_t d2;   // (d, d)
  __device__ __forceinline__ void set(float d) { asm("mov.b64 %0, {%1, %1};" : "=l"(d2) : "r"(__float_as_uint(d))); }
  __device__ __forceinline__ uint32_t pair32(uint32_t m) const {
    float a, b;
    if constexpr (std::is_same<MT, __half>::value) {
      a = __low2float(u32_as_h2(m));
      b = __high2float(u32_as_h2(m));
    } else {
      a = __uint_as_float(m << 16);
      b = __uint_as_float(m & 0xFFFF0000u);
    }
    asm("{.reg .b64 t;\n\tmov.b64 t, {%0, %1};\n\tmul.rn.f32x2 t, t, %2;\n\tmov.b64 {%0, %1}, t;}" : "+f"(a), "+f"(b) : "l"(d2));
    return pack2<ab_t>(a, b);
  }
};
struct Iq3Split {   // d * 256 in two fp16 numbers
  __half2 hi, lo;
  bool wide;
  __device__ __forceinline__ void set(float d) {
    hi = __float2half2_rn(d);
    lo = __float2half2_rn(d - __low2float(hi));
    wide = !(fabsf(d) < 60000.f);
  }
  __device__ __forceinline__ uint32_t pair(uint32_t m) const {
    const __half2 v = u32_as_h2(m);
    return h2_as_u32(__hfma2(v, hi, __hmul2_rn(v, lo)));
  }
};
template <typename ab_t> struct Item128<T_IQ3_XXS, ab_t> {   // half d | u8 qs[64] | per 32 values four 7-bit sign indices and a 4-bit scale; 98 bytes
  static constexpr bool HAVE = true;
  struct State { uint32_t q[8], aux[4]; float dh; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<8>(row + 2 + 32 * ip, wide, s.q);
    lds_row_words<4>(row + 66 + 16 * ip, wide, s.aux);
    s.dh = lds_half_f32(row);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx& cx, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t aux = s.aux[2 * H + u];
      Iq3Scale<__nv_bfloat16, ab_t> g;
      g.set(s.dh * (0.5f + (float)(aux >> 28)) * 0.5f);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const uint32_t w = s.q[4 * H + 2 * u + (l >> 1)], sw = sign_word<T_IQ3_XXS>(cx, (aux >> (7 * l)) & 127u);
        const uint2 a = grid64<T_IQ3_XXS>(cx, byte_of(w, 2 * (l & 1))), b = grid64<T_IQ3_XXS>(cx, byte_of(w, 2 * (l & 1) + 1));
        uint32_t* o = out + 16 * u + 4 * l;
        o[0] = negate(g.pair32(a.x), sign_bits<0>(sw));
        o[1] = negate(g.pair32(a.y), sign_bits<1>(sw));
        o[2] = negate(g.pair32(b.x), sign_bits<2>(sw));
        o[3] = negate(g.pair32(b.y), sign_bits<3>(sw));
      }
    }
  }
};
template <typename ab_t> struct Item128<T_IQ3_S, ab_t> {   // half d | u8 qs[64] | u8 qh[8] | u8 signs[32] | u8 scales[4], 110 bytes
  static constexpr bool HAVE = true;
  struct State { uint32_t q[8], sg[4], qh, sc; float dh; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int, State& s) {
    lds_row_words<8>(row + 2 + 32 * ip, wide, s.q);
    lds_row_words<4>(row + 74 + 16 * ip, wide, s.sg);
    uint32_t w[1];
    lds_words_unaligned<1>(row + 66 + 4 * ip, w);
    s.qh = w[0];
    s.sc = lds16(row + 106 + 2 * ip);
    s.dh = lds_half_f32(row);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx& cx, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t qh = s.qh >> (16 * H + 8 * u), sg = s.sg[2 * H + u];
      constexpr bool SPLIT = std::is_same<ab_t, __half>::value;
      const float d = s.dh * (0.5f + (float)((s.sc >> (8 * H + 4 * u)) & 0xFu)) * (SPLIT ? 128.f : 0.5f);   // (the magnitudes are divided by 256)
      Iq3Scale<ab_t, ab_t> g;
      g.set(d);
      auto go = [&](auto value) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // a word of indices: 16 values
          const uint32_t w = s.q[4 * H + 2 * u + h], top = spread_bits4(qh >> (4 * h));
          const uint2 e[4] = {grid64<T_IQ3_S>(cx, byte_of9<0>(w, top)), grid64<T_IQ3_S>(cx, byte_of9<1>(w, top)),
                              grid64<T_IQ3_S>(cx, byte_of9<2>(w, top)), grid64<T_IQ3_S>(cx, byte_of9<3>(w, top))};
#pragma unroll
          for (int l = 0; l < 2; ++l) {
            const uint32_t sb = byte_of(sg, 2 * h + l);
            uint32_t* o = out + 16 * u + 8 * h + 4 * l;
            o[0] = negate(value(e[2 * l].x), sign_bits8<0>(sb));
            o[1] = negate(value(e[2 * l].y), sign_bits8<1>(sb));
            o[2] = negate(value(e[2 * l + 1].x), sign_bits8<2>(sb));
            o[3] = negate(value(e[2 * l + 1].y), sign_bits8<3>(sb));
          }
        }
      };
      if constexpr (SPLIT) {
        Iq3Split h;
        h.set(d);
        if (!h.wide) {
          go([&](uint32_t m) { return h.pair(m); });
          continue;
        }
      }
      go([&](uint32_t m) { return g.pair32(m); });
    }
  }
};

// ---- the IQ4 formats with fp16 activations: value = round(dl * level), dl in fp32 (at most 17 significant bits) ----
// As IQ3: the level, divided by 128, is 1024 + (level + 128) made by a permute, times 1/128, minus 9 -- exact -- and dl times 128 is split
// in two.  (bf16 has no room for the byte under a power of two: iq4_word.  14336x4096, 48 tokens:
// IQ4_XS 26.2 -> 24.1 us, IQ4_NL 29.7 -> 23.9.)
struct Iq4Group {
  __half2 hi, lo;
  float dl;
  bool big;
  __device__ __forceinline__ void set(float v) {
    dl = v;
    const float d = 128.f * v;
    hi = __float2half2_rn(d);
    lo = __float2half2_rn(d - __low2float(hi));
    big = !(fabsf(d) < 60000.f);
  }
  // a word of indices: values 4i .. 4i + 3 in the low nibbles, 16 + 4i .. in the high ones
  __device__ __forceinline__ void word(uint32_t w, uint32_t* o_lo, uint32_t* o_hi) const {
    if (big) iq4_word<__half>(w, dl, o_lo, o_hi);
    else word16(w, o_lo, o_hi);
  }
  // the 32 values of four words, with one branch
  __device__ __forceinline__ void words(const uint32_t (&w)[4], uint32_t* o) const {
    if (big) {
#pragma unroll
      for (int i = 0; i < 4; ++i) iq4_word<__half>(w[i], dl, o + 2 * i, o + 8 + 2 * i);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) word16(w[i], o + 2 * i, o + 8 + 2 * i);
    }
  }
  __device__ __forceinline__ void word16(uint32_t w, uint32_t* o_lo, uint32_t* o_hi) const {
    const uint32_t q3 = w & 0x77777777u, sel = ((w >> 1) & 0x44444444u) | 0x32103210u;
    const uint32_t a = iq4_levels4(q3, sel), b = iq4_levels4(q3 >> 16, sel >> 16);   // bytes (4i, 16+4i, 4i+1, 17+4i) and (4i+2, ...)
    auto v = [&](uint32_t x) {
      const __half2 m = __hfma2(u32_as_h2(x), __floats2half2_rn(0.0078125f, 0.0078125f), __floats2half2_rn(-9.f, -9.f));
      return h2_as_u32(__hfma2(m, hi, __hmul2_rn(m, lo)));
    };
    o_lo[0] = v(__byte_perm(a, 0x64646464u, 0x4240));
    o_lo[1] = v(__byte_perm(b, 0x64646464u, 0x4240));
    o_hi[0] = v(__byte_perm(a, 0x64646464u, 0x4341));
    o_hi[1] = v(__byte_perm(b, 0x64646464u, 0x4341));
  }
};
template <> struct Item128<T_IQ4_XS, __half> {   // half d | u16 scales_h | u8 scales_l[4] | u8 qs[128], 136 bytes (8-byte aligned)
  static constexpr bool HAVE = true;
  struct State { float d; uint32_t lo, hi; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool, int, State& s) {
    const uint2 h = lds64(row);
    s.d = __half2float(__ushort_as_half((unsigned short)(h.x & 0xFFFFu)));
    s.hi = h.x >> (16 + 8 * ip);
    s.lo = h.y >> (16 * ip);
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t row, int ip, bool, const DecodeCtx&, const State& s, uint32_t (&out)[32]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int ib = 2 * H + u;
      const uint2 a = lds64(row + 8 + 64 * ip + 16 * ib), b = lds64(row + 16 + 64 * ip + 16 * ib);
      Iq4Group g;
      g.set(s.d * (float)((int)(((s.lo >> (4 * ib)) & 0xFu) | (((s.hi >> (2 * ib)) & 3u) << 4)) - 32));
      uint32_t* o = out + 16 * u;
      g.word(a.x, o, o + 8);
      g.word(a.y, o + 2, o + 10);
      g.word(b.x, o + 4, o + 12);
      g.word(b.y, o + 6, o + 14);
    }
  }
};
// IQ4_NL: the words of both stages at once and one branch a block.  (Read by the stage, with a branch a word, the decoder held the few A slots of the
// largest tiles for too long: 384 tokens of 14336x4096 44.3 us against 40.2 with unit decoders, now 39.2; 17 tokens 26.9 -> 23.5.  The unit
// decoder that bf16 had fetched every block's bytes by itself: 384 tokens 40.9 -> 38.9, 17 tokens 29.4 -> 26.4, same arithmetic.)
template <typename ab_t> struct Item128<T_IQ4_NL, ab_t> {   // blocks of 18 bytes: half d | u8 qs[16]
  static constexpr bool HAVE = true;
  struct State { uint32_t w[18]; int left; };
  static __device__ __forceinline__ void begin(uint32_t row, int ip, bool wide, int left, State& s) {
    lds_row_words<18>(row + 72 * ip, wide, s.w);
    s.left = left;
  }
  template <int H> static __device__ __forceinline__ void stage(uint32_t, int, bool, const DecodeCtx&, const State& s, uint32_t (&out)[32]) {
    const uint32_t* w = s.w + 9 * H;
#pragma unroll
    for (int u = 0; u < 2; ++u) {   // the second block starts 18 bytes on: its d in the upper half of word four
      const float d = __half2float(__ushort_as_half((unsigned short)(u ? w[4] >> 16 : w[0] & 0xFFFFu)));
      const float dl = 2 * H + u < s.left ? d : 0.f;   // (beyond the row: what follows it)
      uint32_t q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = u ? w[5 + i] : __funnelshift_r(w[i], w[i + 1], 16);
      if constexpr (std::is_same<ab_t, __half>::value) {
        Iq4Group g;
        g.set(dl);
        g.words(q, out + 16 * u);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) iq4_word<ab_t>(q[i], dl, out + 16 * u + 2 * i, out + 16 * u + 8 + 2 * i);
      }
    }
  }
};

}  // namespace gguf_b200
