// Weight decoders of the small-batch kernel (smallm.cu): one 32-value block of two weight rows as the A
// fragment of an 8-bit tensor instruction.
//
// The lane (g, t) = (lane / 4, lane % 4) holds two words, eight codes, of row g (and, by a second call, of
// row g + 8); which eight of the 32 is free as long as the activations follow (the contraction does not
// care), so each format takes the order its bytes already have (`ORDER`, see quantize_frag_kernel):
//   0  words (4t .. 4t+3) and (16+4t ..)       nibble formats whose halves are 16 values apart, and
//                                              formats with a scale per 16 values
//   1  words (8t .. 8t+3) and (8t+4 ..)        formats with 32 consecutive bytes or 8-value code-book entries
//   2  the bytes of order 0 interleaved: (4t, 16+4t, 4t+1, 17+4t) and (4t+2, 18+4t, 4t+3, 19+4t)
//                                              what two byte-permutes make of a word of 4-bit IQ4 indices
//
// With isum = sum over the block of code * q8, a block adds to the result
//   KIND 0:  s * d8 * isum
//   KIND 2:  half(d * d8) * isum + half(m * s8)                  (Q4_1, Q5_1: products rounded as the reference does)
//   KIND 3:  d8 * (s * isum(first 16) + m * isum(last 16))       (a scale per 16 values: two k = 16 instructions)
//   KIND 4:  d8 * (s * isum + m * msum), msum from a second instruction on the words v0, v1 (Q2_K)
// and, for the formats with a minimum or an offset (MINS), the chunk as a whole adds mf * sum over its blocks of min * s8: a
// small product of its own, min (exact in tf32: an integer, or one fp16 number) against s8 in two tf32 parts, which takes two
// tensor instructions per chunk and tile instead of four multiply-adds per block.
// These are the formulas of the reference's vec_dot_*_q8_1 (vecdotq.cuh:493-509, 852-1048, 1159-1202, 1417-1441, 1531-1812).
// Codes are bytes; where the code times a sub-block scale, or the code shifted left, still fits a byte that is what the tensor
// core sees, which saves work on its result.  All of it is exact integer arithmetic.
#pragma once

#include "common.cuh"
#include "tables.cuh"

namespace gguf_b200 {

// Loads are asm without `volatile`: pure functions of the address, so that blocks that read the same words share one load.
// Every address derives from sm_fresh(), a volatile statement behind the barrier wait.
__device__ __forceinline__ uint32_t sm_fresh(uint32_t a) {
  uint32_t r;
  asm volatile("mov.u32 %0, %1;" : "=r"(r) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ uint32_t sl32(uint32_t a) { uint32_t v; asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 sl64(uint32_t a) { uint2 v; asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint4 sl128(uint32_t a) { uint4 v; asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t sl16(uint32_t a) { unsigned short v; asm("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t sl8(uint32_t a) { uint32_t v; asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ float slh(uint32_t a) { return __half2float(__ushort_as_half((unsigned short)sl16(a))); }
__device__ __forceinline__ float h2f(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)(bits & 0xFFFFu))); }
// N words from a 2-byte aligned address
template <int N> __device__ __forceinline__ void slw(uint32_t a, uint32_t (&w)[N]) {
  const uint32_t al = a & ~3u, sh = (a & 3u) * 8u;
  uint32_t r[N + 1];
#pragma unroll
  for (int i = 0; i <= N; ++i) r[i] = sl32(al + 4u * i);
#pragma unroll
  for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(r[i], r[i + 1], sh);
}
__device__ __forceinline__ uint32_t slw1(uint32_t a) { uint32_t w[1]; slw<1>(a, w); return w[0]; }

// ... from a + off, `a` a multiple of four.  KNOWN: so is the row's start, and off, a constant where this is called, says how
// the words lie -- no address arithmetic, no second load where they are aligned.
template <bool KNOWN, int N> __device__ __forceinline__ void slwo(uint32_t a, int off, uint32_t (&w)[N]) {
  if constexpr (!KNOWN) {
    slw<N>(a + off, w);
  } else if ((off & 3) == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = sl32(a + off + 4 * i);
  } else {
    uint32_t r[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) r[i] = sl32(a + (off & ~3) + 4 * i);
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = __byte_perm(r[i], r[i + 1], 0x5432);   // (offsets are even)
  }
}
template <bool KNOWN> __device__ __forceinline__ uint32_t slwo1(uint32_t a, int off) { uint32_t w[1]; slwo<KNOWN, 1>(a, off, w); return w[0]; }

struct SmBlk {
  uint32_t w0, w1;     // codes
  uint32_t v0, v1;     // KIND 4: minima
  float s, m;
  uint32_t dm;         // KIND 2: {d, m}
};
struct SmNone {};

// An unsigned byte as a float without a conversion instruction: byte k of w under the exponent of 2^23 is 2^23 + byte.
__device__ __forceinline__ float sm_byte_2p23(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | k)); }
struct SmScale {       // x * byte = x * (2^23 + byte) - x * 2^23 in one fused multiply-add (exact product and offset, one rounding)
  float x, off;
  __device__ __forceinline__ void set(float v) { x = v; off = -8388608.f * v; }
  __device__ __forceinline__ float at(uint32_t w, int k) const { return fmaf(x, sm_byte_2p23(w, k), off); }
};
// x * (byte - bias)
__device__ __forceinline__ float sm_biased(float x, uint32_t w, int k, float bias) { return x * (sm_byte_2p23(w, k) - (8388608.f + bias)); }
// byte k of w, k known at run time only, as a float
__device__ __forceinline__ float sm_byte(uint32_t w, int k) { return (float)((w >> (8 * k)) & 0xFFu); }

// four sign bits -> the bytes of g negated where the bit is set (g >= 1 per byte, so no carry leaves a byte)
__device__ __forceinline__ uint32_t sm_apply_signs(uint32_t g, uint32_t nib) {
  const uint32_t s01 = ((nib & 0xFu) * 0x00204081u) & 0x01010101u;
  return (g ^ (s01 * 255u)) + s01;
}
// seven sign bits and the eighth that makes the number of negative signs even
__device__ __forceinline__ uint32_t sm_signs7(uint32_t s7) { return s7 | ((__popc(s7) & 1u) << 7); }
__device__ __forceinline__ uint32_t sm_spread4(uint32_t x) { return ((x & 0xFu) * 0x02040810u) & 0x10101010u; }   // bit j -> bit 4 of byte j

// rp: shared address of the row's chunk (256 values); j: block 0..7 of the chunk; t: lane % 4; tab: shared code book.
// U8: the codes are unsigned bytes.  MINS: mins(rp, row, t, nb, a) gives the minima of the blocks t and t + 4 (0 for blocks
// from nb on) and returns the row's factor.
template <int TYPE> struct SmDec;
// the formats of 32-value blocks: rows of whole chunks of which start on 16-byte boundaries (block<KNOWN>)
template <int TYPE> __host__ __device__ constexpr bool sm_can_be_whole() {
  return TYPE == T_Q4_0 || TYPE == T_Q4_1 || TYPE == T_Q5_0 || TYPE == T_Q5_1 || TYPE == T_Q8_0 || TYPE == T_IQ4_NL;
}

template <> struct SmDec<T_Q4_0> {
  static constexpr int ORDER = 0, KIND = 0;
  static constexpr bool U8 = true, MINS = true;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  static __device__ __forceinline__ float mins(uint32_t rp, const Row&, int t, int nb, float (&a)[2]) {
    a[0] = t < nb ? slh(rp + 18 * t) : 0.f;
    a[1] = t + 4 < nb ? slh(rp + 18 * (t + 4)) : 0.f;
    return -8.f;
  }
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    const uint32_t q = slwo1<KNOWN>(rp + 4 * t, 18 * j + 2);
    b.w0 = q & 0x0F0F0F0Fu;
    b.w1 = (q >> 4) & 0x0F0F0F0Fu;
    b.s = slh(rp + 18 * j);
  }
};
template <> struct SmDec<T_Q4_1> {
  static constexpr int ORDER = 0, KIND = 2;
  static constexpr bool U8 = true, MINS = false;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    const uint32_t q = sl32(rp + 20 * j + 4 + 4 * t);
    b.w0 = q & 0x0F0F0F0Fu;
    b.w1 = (q >> 4) & 0x0F0F0F0Fu;
    b.dm = sl32(rp + 20 * j);
  }
};
template <> struct SmDec<T_Q5_0> {
  static constexpr int ORDER = 0, KIND = 0;
  static constexpr bool U8 = true, MINS = true;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  static __device__ __forceinline__ float mins(uint32_t rp, const Row&, int t, int nb, float (&a)[2]) {
    a[0] = t < nb ? slh(rp + 22 * t) : 0.f;
    a[1] = t + 4 < nb ? slh(rp + 22 * (t + 4)) : 0.f;
    return -16.f;
  }
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    const uint32_t qh = slwo1<KNOWN>(rp, 22 * j + 2), q = slwo1<KNOWN>(rp + 4 * t, 22 * j + 6);
    b.w0 = (q & 0x0F0F0F0Fu) | sm_spread4(qh >> (4 * t));
    b.w1 = ((q >> 4) & 0x0F0F0F0Fu) | sm_spread4(qh >> (16 + 4 * t));
    b.s = slh(rp + 22 * j);
  }
};
template <> struct SmDec<T_Q5_1> {
  static constexpr int ORDER = 0, KIND = 2;
  static constexpr bool U8 = true, MINS = false;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    const uint2 h = sl64(rp + 24 * j);
    const uint32_t q = sl32(rp + 24 * j + 8 + 4 * t);
    b.w0 = (q & 0x0F0F0F0Fu) | sm_spread4(h.y >> (4 * t));
    b.w1 = ((q >> 4) & 0x0F0F0F0Fu) | sm_spread4(h.y >> (16 + 4 * t));
    b.dm = h.x;
  }
};
template <> struct SmDec<T_Q8_0> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    uint32_t w[2];
    slwo<KNOWN, 2>(rp + 8 * t, 34 * j + 2, w);
    b.w0 = w[0];
    b.w1 = w[1];
    b.s = slh(rp + 34 * j);
  }
};
// the 6-bit scales and minima of a Q4_K / Q5_K super-block, a byte each: [0] sub-blocks 0-3, [1] sub-blocks 4-7
struct SmScales {
  SmScale d, dh;       // dh: d / 16, for the codes that stay in the high nibbles
  float dmin;
  uint32_t sc[2], mn[2];
  __device__ __forceinline__ void load(uint32_t rp) {
    const uint4 h = sl128(rp);
    const float v = h2f(h.x);
    d.set(v);
    dh.set(v * 0.0625f);
    dmin = -h2f(h.x >> 16);
    sc[0] = h.y & 0x3F3F3F3Fu;
    mn[0] = h.z & 0x3F3F3F3Fu;
    sc[1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    mn[1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
  }
  __device__ __forceinline__ float mins(int t, float (&a)[2]) const {
    a[0] = sm_byte(mn[0], t);
    a[1] = sm_byte(mn[1], t);
    return dmin;
  }
};
template <> struct SmDec<T_Q4_K> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = true, MINS = true;
  using Row = SmScales;
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) { r.load(rp); }
  static __device__ __forceinline__ float mins(uint32_t, const Row& r, int t, int, float (&a)[2]) { return r.mins(t, a); }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    const uint2 q = sl64(rp + 16 + 32 * (j >> 1) + 8 * t);
    const uint32_t mask = j & 1 ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
    b.w0 = q.x & mask;
    b.w1 = q.y & mask;
    b.s = (j & 1 ? r.dh : r.d).at(r.sc[j >> 2], j & 3);
  }
};
template <> struct SmDec<T_Q5_K> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = true, MINS = true;
  using Row = SmScales;
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) { r.load(rp); }
  static __device__ __forceinline__ float mins(uint32_t, const Row& r, int t, int, float (&a)[2]) { return r.mins(t, a); }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    const uint2 h = sl64(rp + 16 + 8 * t), q = sl64(rp + 48 + 32 * (j >> 1) + 8 * t);
    b.w0 = ((q.x >> (4 * (j & 1))) & 0x0F0F0F0Fu) | ((j < 4 ? h.x << (4 - j) : h.x >> (j - 4)) & 0x10101010u);
    b.w1 = ((q.y >> (4 * (j & 1))) & 0x0F0F0F0Fu) | ((j < 4 ? h.y << (4 - j) : h.y >> (j - 4)) & 0x10101010u);
    b.s = r.d.at(r.sc[j >> 2], j & 3);
  }
};
// Q6_K: the byte is 4 * (code - 32): the code in bits 2-7 with the top bit flipped
template <> struct SmDec<T_Q6_K> {
  static constexpr int ORDER = 0, KIND = 3;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t sc[4]; };   // sc: the int8 scales plus 128
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.d = 0.25f * slh(rp + 208);
    slw<4>(rp + 192, r.sc);
#pragma unroll
    for (int i = 0; i < 4; ++i) r.sc[i] ^= 0x80808080u;
  }
  static __device__ __forceinline__ uint32_t word(uint32_t l, uint32_t h, int q) {
    const uint32_t lo = q >> 1 ? (l >> 2) & 0x3C3C3C3Cu : (l << 2) & 0x3C3C3C3Cu;
    const uint32_t hi = q < 3 ? h << (6 - 2 * q) : h;
    return lo | ((hi & 0xC0C0C0C0u) ^ 0x80808080u);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    const int ip = j >> 2, q = j & 3;
    const uint32_t ql = rp + 64 * ip + 32 * (q & 1) + 4 * t, qh = rp + 128 + 32 * ip + 4 * t;
    b.w0 = word(slw1(ql), slw1(qh), q);
    b.w1 = word(slw1(ql + 16), slw1(qh + 16), q);
    b.s = sm_biased(r.d, r.sc[j >> 1], 2 * (j & 1), 128.f);
    b.m = sm_biased(r.d, r.sc[j >> 1], 2 * (j & 1) + 1, 128.f);
  }
};
// Q2_K: the byte is scale * code (at most 45), the minima go through an instruction of their own
template <> struct SmDec<T_Q2_K> {
  static constexpr int ORDER = 0, KIND = 4;
  static constexpr bool U8 = true, MINS = false;
  struct Row { float d, dmin; uint32_t sc[4]; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    const uint32_t dm = sl32(rp + 80);
    r.d = h2f(dm);
    r.dmin = -h2f(dm >> 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) r.sc[i] = sl32(rp + 4 * i);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    const uint32_t q = rp + 16 + 32 * (j >> 2) + 4 * t;
    const uint32_t s2 = r.sc[j >> 1] >> (16 * (j & 1));
    b.w0 = ((sl32(q) >> (2 * (j & 3))) & 0x03030303u) * (s2 & 0xFu);
    b.w1 = ((sl32(q + 16) >> (2 * (j & 3))) & 0x03030303u) * ((s2 >> 8) & 0xFu);
    b.v0 = ((s2 >> 4) & 0xFu) * 0x01010101u;
    b.v1 = ((s2 >> 12) & 0xFu) * 0x01010101u;
    b.s = r.d;
    b.m = r.dmin;
  }
};
// Q3_K: the byte is -(scale - 32) * (code - 4), which reaches -128 but never +128
template <> struct SmDec<T_Q3_K> {
  static constexpr int ORDER = 0, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t sc[4]; };   // sc: 6-bit scales, sub-blocks 4i .. 4i + 3
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.d = -slh(rp + 108);
    uint32_t w[3];
    slw<3>(rp + 96, w);
    r.sc[0] = (w[0] & 0x0F0F0F0Fu) | ((w[2] << 4) & 0x30303030u);
    r.sc[1] = (w[1] & 0x0F0F0F0Fu) | ((w[2] << 2) & 0x30303030u);
    r.sc[2] = ((w[0] >> 4) & 0x0F0F0F0Fu) | (w[2] & 0x30303030u);
    r.sc[3] = ((w[1] >> 4) & 0x0F0F0F0Fu) | ((w[2] >> 2) & 0x30303030u);
  }
  static __device__ __forceinline__ uint32_t word(uint32_t q, uint32_t h, int j, uint32_t sc6) {
    const uint32_t c = ((q >> (2 * (j & 3))) & 0x03030303u) | (((h >> j) & 0x01010101u) << 2);   // code 0..7
    const uint32_t k = (32u - sc6) & 0xFFu;                                                       // -(scale), modulo 256
    const uint32_t off = ((sc6 - 32u) * 4u & 0xFFu) * 0x00010001u;                                // k * (c - 4) = k * c + 4 * scale
    const uint32_t lo = (c & 0x00FF00FFu) * k + off, hi = ((c >> 8) & 0x00FF00FFu) * k + off;     // 16-bit lanes: no carries
    return __byte_perm(lo, hi, 0x6240);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    const uint32_t q = rp + 32 + 32 * (j >> 2) + 4 * t, h = rp + 4 * t;
    const uint32_t s2 = r.sc[j >> 1] >> (16 * (j & 1));
    b.w0 = word(slw1(q), slw1(h), j, s2 & 0xFFu);
    b.w1 = word(slw1(q + 16), slw1(h + 16), j, (s2 >> 8) & 0xFFu);
    b.s = r.d;
  }
};
// the sixteen IQ4 levels in four registers: two byte-permutes look four indices up in a half of the table each (the word's
// nibbles are the selectors), a third takes the half that the index's top bit names
__device__ __forceinline__ uint32_t sm_iq4(uint32_t q3, uint32_t sel) {
  // levels -127 -104 -83 -65 | -49 -35 -22 -10 | 1 13 25 38 | 53 69 89 113
  return __byte_perm(__byte_perm(0xBFAD9881u, 0xF6EADDCFu, q3), __byte_perm(0x26190D01u, 0x71594535u, q3), sel);
}
__device__ __forceinline__ void sm_iq4_words(uint32_t q, uint32_t& w0, uint32_t& w1) {
  const uint32_t q3 = q & 0x77777777u, sel = ((q & 0x88888888u) >> 1) | 0x32103210u;
  w0 = sm_iq4(q3, sel);
  w1 = sm_iq4(q3 >> 16, sel >> 16);
}
template <> struct SmDec<T_IQ4_NL> {
  static constexpr int ORDER = 2, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  using Row = SmNone;
  static __device__ __forceinline__ void head(uint32_t, Row&) {}
  template <bool KNOWN> static __device__ __forceinline__ void block(uint32_t rp, const Row&, int j, int t, uint32_t, SmBlk& b) {
    sm_iq4_words(slwo1<KNOWN>(rp + 4 * t, 18 * j + 2), b.w0, b.w1);
    b.s = slh(rp + 18 * j);
  }
};
template <> struct SmDec<T_IQ4_XS> {
  static constexpr int ORDER = 2, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t ls[2]; };   // 6-bit scales, a byte each: [0] even blocks, [1] odd blocks
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    const uint2 h = sl64(rp);
    r.d = h2f(h.x);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t x = h.x >> (16 + 2 * i);   // two high bits of the blocks i, i + 2, i + 4, i + 6 at bits 0, 4, 8, 12
      r.ls[i] = ((h.y >> (4 * i)) & 0x0F0F0F0Fu) | ((x & 0x3u) << 4) | ((x & 0x30u) << 8) | ((x & 0x300u) << 12) | ((x & 0x3000u) << 16);
    }
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t, SmBlk& b) {
    sm_iq4_words(sl32(rp + 8 + 16 * j + 4 * t), b.w0, b.w1);
    b.s = sm_biased(r.d, r.ls[j & 1], j >> 1, 32.f);
  }
};
// code-book formats: tab holds the grid; a scale (2 * n + 1) with n a 4-bit field
__device__ __forceinline__ float sm_odd_scale(float d, uint32_t n) { return fmaf(d + d, (float)n, d); }   // exact: d has 11 bits
template <> struct SmDec<T_IQ2_XXS> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) { r.d = 0.125f * slh(rp); }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    uint32_t q[2];
    slw<2>(rp + 2 + 8 * j, q);
    const uint2 g = sl64(tab + 8u * ((q[0] >> (8 * t)) & 0xFFu));
    const uint32_t s = sm_signs7((q[1] >> (7 * t)) & 127u);
    b.w0 = sm_apply_signs(g.x, s);
    b.w1 = sm_apply_signs(g.y, s >> 4);
    b.s = sm_odd_scale(r.d, q[1] >> 28);
  }
};
template <> struct SmDec<T_IQ2_XS> {   // two 8-value entries per scale: lane t takes one word of the entries t/2 and 2 + t/2
  static constexpr int ORDER = 0, KIND = 3;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t sc[2]; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.d = 0.125f * slh(rp);
    slw<2>(rp + 66, r.sc);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const uint32_t q = rp + 2 + 8 * j + 2 * (t >> 1), e0 = sl16(q), e1 = sl16(q + 4);
    b.w0 = sm_apply_signs(sl32(tab + 8u * (e0 & 511u) + 4u * (t & 1)), sm_signs7(e0 >> 9) >> (4 * (t & 1)));
    b.w1 = sm_apply_signs(sl32(tab + 8u * (e1 & 511u) + 4u * (t & 1)), sm_signs7(e1 >> 9) >> (4 * (t & 1)));
    const uint32_t sc = r.sc[j >> 2] >> (8 * (j & 3));
    b.s = sm_odd_scale(r.d, sc & 0xFu);
    b.m = sm_odd_scale(r.d, (sc >> 4) & 0xFu);
  }
};
template <> struct SmDec<T_IQ2_S> {
  static constexpr int ORDER = 0, KIND = 3;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t qh[2], sc[2]; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.d = 0.125f * slh(rp);
    slw<2>(rp + 66, r.qh);
    slw<2>(rp + 74, r.sc);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const int l = t >> 1;
    const uint32_t q = slw1(rp + 2 + 4 * j), sg = slw1(rp + 34 + 4 * j), qh = (r.qh[j >> 2] >> (8 * (j & 3))) & 0xFFu;
    const uint32_t e0 = ((q >> (8 * l)) & 0xFFu) | ((qh << (8 - 2 * l)) & 0x300u), e1 = ((q >> (16 + 8 * l)) & 0xFFu) | ((qh << (4 - 2 * l)) & 0x300u);
    b.w0 = sm_apply_signs(sl32(tab + 8u * e0 + 4u * (t & 1)), sg >> (8 * l + 4 * (t & 1)));
    b.w1 = sm_apply_signs(sl32(tab + 8u * e1 + 4u * (t & 1)), sg >> (16 + 8 * l + 4 * (t & 1)));
    const uint32_t sc = r.sc[j >> 2] >> (8 * (j & 3));
    b.s = sm_odd_scale(r.d, sc & 0xFu);
    b.m = sm_odd_scale(r.d, (sc >> 4) & 0xFu);
  }
};
template <> struct SmDec<T_IQ3_XXS> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) { r.d = 0.25f * slh(rp); }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const uint32_t e = sl16(rp + 2 + 8 * j + 2 * t), aux = slw1(rp + 66 + 4 * j);
    const uint32_t s = sm_signs7((aux >> (7 * t)) & 127u);
    b.w0 = sm_apply_signs(sl32(tab + 4u * (e & 0xFFu)), s);
    b.w1 = sm_apply_signs(sl32(tab + 4u * (e >> 8)), s >> 4);
    b.s = sm_odd_scale(r.d, aux >> 28);
  }
};
template <> struct SmDec<T_IQ3_S> {
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint32_t qh[2], sc; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.d = 0.25f * slh(rp);
    slw<2>(rp + 66, r.qh);
    r.sc = slw1(rp + 106);
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const uint32_t e = sl16(rp + 2 + 8 * j + 2 * t), sg = sl8(rp + 74 + 4 * j + t), qh = (r.qh[j >> 2] >> (8 * (j & 3))) & 0xFFu;
    b.w0 = sm_apply_signs(sl32(tab + 4u * ((e & 0xFFu) | ((qh << (8 - 2 * t)) & 256u))), sg);
    b.w1 = sm_apply_signs(sl32(tab + 4u * ((e >> 8) | ((qh << (7 - 2 * t)) & 256u))), sg >> 4);
    b.s = sm_odd_scale(r.d, (r.sc >> (4 * j)) & 0xFu);
  }
};
template <> struct SmDec<T_IQ1_S> {   // the offset (-1 +- 1/8 times the block's scale) meets the sum of the inputs
  static constexpr int ORDER = 1, KIND = 0;
  static constexpr bool U8 = true, MINS = true;
  struct Row { float d; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) { r.d = slh(rp); }
  static __device__ __forceinline__ float mins(uint32_t rp, const Row& r, int t, int, float (&a)[2]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t qh = sl16(rp + 34 + 2 * (t + 4 * h));
      a[h] = (float)((int)(2u * ((qh >> 12) & 7u) + 1u) * (qh & 0x8000u ? -9 : -7));
    }
    return 0.125f * r.d;
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const uint32_t q = sl8(rp + 2 + 4 * j + t), qh = sl16(rp + 34 + 2 * j);
    const uint32_t g = sl32(tab + 4u * (q | (((qh >> (3 * t)) & 7u) << 8)));
    b.w0 = g & 0x0F0F0F0Fu;
    b.w1 = (g >> 4) & 0x0F0F0F0Fu;
    b.s = sm_odd_scale(r.d, (qh >> 12) & 7u);
  }
};
template <> struct SmDec<T_IQ1_M> {   // the byte is 8 * (code + offset): codes 0, 1, 2, offsets -1 +- 1/8
  static constexpr int ORDER = 0, KIND = 3;
  static constexpr bool U8 = false, MINS = false;
  struct Row { float d; uint2 sc; };
  static __device__ __forceinline__ void head(uint32_t rp, Row& r) {
    r.sc = sl64(rp + 48);
    r.d = 0.125f * h2f(((r.sc.x >> 12) & 0x000Fu) | ((r.sc.x >> 24) & 0x00F0u) | ((r.sc.y >> 4) & 0x0F00u) | ((r.sc.y >> 16) & 0xF000u));
  }
  static __device__ __forceinline__ uint32_t word(uint32_t g, uint32_t neg, int half) {
    const uint32_t c = (g >> (4 * half)) & 0x0F0F0F0Fu;
    return (8u * c + (neg ? 0x77777777u : 0x79797979u)) ^ 0x80808080u;   // 8c - 9 or 8c - 7, a byte each
  }
  static __device__ __forceinline__ void block(uint32_t rp, const Row& r, int j, int t, uint32_t tab, SmBlk& b) {
    const int l = t >> 1;
    const uint32_t q = sl32(rp + 4 * j), qh = sl16(rp + 32 + 2 * j);
    const uint32_t h0 = qh >> (4 * l), h1 = qh >> (8 + 4 * l);
    b.w0 = word(sl32(tab + 4u * (((q >> (8 * l)) & 0xFFu) | ((h0 & 7u) << 8))), h0 & 8u, t & 1);
    b.w1 = word(sl32(tab + 4u * (((q >> (16 + 8 * l)) & 0xFFu) | ((h1 & 7u) << 8))), h1 & 8u, t & 1);
    const uint32_t s2 = ((j & 4) ? r.sc.y : r.sc.x) >> (16 * ((j >> 1) & 1) + 6 * (j & 1));
    b.s = sm_odd_scale(r.d, s2 & 7u);
    b.m = sm_odd_scale(r.d, (s2 >> 3) & 7u);
  }
};

// code books: bytes in shared memory
template <int TYPE> __host__ __device__ constexpr int sm_table_bytes() {
  return TYPE == T_IQ2_XXS ? 2048 : TYPE == T_IQ2_XS ? 4096 : TYPE == T_IQ2_S ? 8192 : TYPE == T_IQ3_XXS ? 1024 : TYPE == T_IQ3_S ? 2048
         : (TYPE == T_IQ1_S || TYPE == T_IQ1_M) ? 8192 : 0;
}
template <int TYPE> __device__ __forceinline__ const uint32_t* sm_table_source() {
  if constexpr (TYPE == T_IQ2_XXS) return reinterpret_cast<const uint32_t*>(d_iq2xxs_grid);
  if constexpr (TYPE == T_IQ2_XS) return reinterpret_cast<const uint32_t*>(d_iq2xs_grid);
  if constexpr (TYPE == T_IQ2_S) return reinterpret_cast<const uint32_t*>(d_iq2s_grid);
  if constexpr (TYPE == T_IQ3_XXS) return reinterpret_cast<const uint32_t*>(d_iq3xxs_grid);
  if constexpr (TYPE == T_IQ3_S) return reinterpret_cast<const uint32_t*>(d_iq3s_grid);
  if constexpr (TYPE == T_IQ1_S || TYPE == T_IQ1_M) return reinterpret_cast<const uint32_t*>(d_iq1s_grid);
  return nullptr;
}
// what follows the {d8} pairs of a block in the activation tiles: KIND 2 keeps {d8, s8}, the others {d8, -1.5 * 2^23 * d8}
inline bool sm_pairs_with_sum(int type) { return type == T_Q4_1 || type == T_Q5_1; }
inline int sm_order(int type) {
  switch (type) {
    case T_Q8_0: case T_Q4_K: case T_Q5_K: case T_IQ2_XXS: case T_IQ3_XXS: case T_IQ3_S: case T_IQ1_S: return 1;
    case T_IQ4_NL: case T_IQ4_XS: return 2;
  }
  return 0;
}

}  // namespace gguf_b200
