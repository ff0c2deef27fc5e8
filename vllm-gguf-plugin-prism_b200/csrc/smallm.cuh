// Kernel of the small-batch product (see smallm.cu, which also explains the layout); instantiated by smallm_inst_*.cu.
#pragma once

#include "kernels.h"
#include "raw_stream.cuh"
#include "smallm_decode.cuh"

namespace gguf_b200 {

constexpr int SM_WARPS = 8;                         // consumer warps, 16 rows each
constexpr int SM_THREADS = (SM_WARPS + 1) * 32;     // + one warp that issues the copies
// an activation tile, one chunk of 256 values of eight columns: codes, the scale pairs of every block and column, and s8 as tf32
// fragments (high and low part, blocks t and t + 4 of column g)
constexpr int SM_CODE_BYTES = 2048, SM_PAIR_BYTES = 512, SM_SUM_BYTES = 512, SM_TILE_BYTES = SM_CODE_BYTES + SM_PAIR_BYTES + SM_SUM_BYTES;
constexpr int SM_MAX_STAGES = 8;

struct SmParams {
  RawPlan raw;
  const uint8_t* w;
  int64_t w_bytes;
  const uint8_t* x;       // activation tiles [chunk][column tile]
  void* y;
  int64_t ldy;            // elements between output rows
  int dtype;
  int n, m;               // weight rows, columns (tokens)
  int nblk, nc, rt;       // 32-value blocks, chunks, row tiles of a row / matrix
  int tiles;              // column tiles in x
  int stages, stage_bytes;
  int ahead;              // stages asked for and not there yet, at most
  float* part;            // partial tiles, two slots per CTA
  int* counter;           // arrivals per output tile, zero at the start
  int* status;
  // MoE (passes != null): pass p works on the matrix of expert passes[p].x for the column tiles passes[p].y .. + passes[p].z
  const int4* passes;
  const int32_t* n_passes;
  const int32_t* sorted;  // output row of every column (>= rows_out: padding)
  int rows_out;
  const float* row_scale; // routing weight of every output row, or null
};

template <bool U8>
__device__ __forceinline__ void sm_mma32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int init) {
  if constexpr (U8)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(init));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(init));
}
__device__ __forceinline__ void sm_mma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, int init) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5},{%6},{%7,%7,%7,%7};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a0), "r"(a1), "r"(b0), "r"(init));
}
__device__ __forceinline__ void sm_mma_tf32(float (&c)[4], const float (&lo)[2], const float (&hi)[2], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(__float_as_uint(lo[0])), "r"(__float_as_uint(hi[0])), "r"(__float_as_uint(lo[1])), "r"(__float_as_uint(hi[1])), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __half2 sm_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// One block (32 values) of the warp's 16 rows against one column tile: acc[0..1] row g, columns 2t, 2t+1; acc[2..3] row g + 8.
// The accumulator of the integer product starts at the bit pattern of 1.5 * 2^23: the result, read as a float, is that number
// plus the sum (exact below 2^22), so no conversion instruction is needed, and the fused multiply-add that scales it by d8
// takes the offset out exactly (d8 has 11 significant bits, the offset two: their product is exact, and comes with the tile).
constexpr int SM_MAGIC = 0x4B400000;
constexpr float SM_MAGIC_F = 12582912.f;
template <int KIND, bool U8>
__device__ __forceinline__ void sm_block(float (&acc)[4], const SmBlk& lo, const SmBlk& hi, uint2 b, float4 dp) {
  // dp: the pair of column 2t, the pair of column 2t + 1
  int c[4];
  auto add = [&](const int (&v)[4], float slo, float shi) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      acc[i] = fmaf(fmaf(__int_as_float(v[i]), i & 1 ? dp.z : dp.x, i & 1 ? dp.w : dp.y), i < 2 ? slo : shi, acc[i]);
  };
  if constexpr (KIND == 3) {
    sm_mma16(c, lo.w0, hi.w0, b.x, SM_MAGIC);
    add(c, lo.s, hi.s);
    sm_mma16(c, lo.w1, hi.w1, b.y, SM_MAGIC);
    add(c, lo.m, hi.m);
  } else {
    sm_mma32<U8>(c, lo.w0, hi.w0, lo.w1, hi.w1, b.x, b.y, SM_MAGIC);
    if constexpr (KIND == 2) {
      const __half2 d2 = __floats2half2_rn(dp.x, dp.z), s2 = __floats2half2_rn(dp.y, dp.w);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t dm = r ? hi.dm : lo.dm;
        const float2 p = __half22float2(__hmul2_rn(sm_h2(__byte_perm(dm, 0u, 0x1010)), d2));
        const float2 q = __half22float2(__hmul2_rn(sm_h2(__byte_perm(dm, 0u, 0x3232)), s2));
        acc[2 * r] += fmaf(__int_as_float(c[2 * r]) - SM_MAGIC_F, p.x, q.x);
        acc[2 * r + 1] += fmaf(__int_as_float(c[2 * r + 1]) - SM_MAGIC_F, p.y, q.y);
      }
    } else {
      add(c, lo.s, hi.s);
      if constexpr (KIND == 4) {
        sm_mma32<U8>(c, lo.v0, hi.v0, lo.v1, hi.v1, b.x, b.y, SM_MAGIC);
        add(c, lo.m, hi.m);
      }
    }
  }
}

template <typename T> __device__ __forceinline__ void sm_store(const SmParams& p, int64_t orow, int n, float v, float scale) {
  T o = from_float<T>(v);
  // routing weight applied as the reference applies it: to the rounded value, rounded again
  if (p.row_scale) o = from_float<T>(to_float<T>(o) * scale);
  static_cast<T*>(p.y)[orow * p.ldy + n] = o;
}

// WHOLE: rows of whole chunks in dense stages: every row and chunk starts on a 16-byte boundary and no chunk is cut short.
// (MoE step of eight tokens, 64 experts of Q4_0: 65 -> 41 instructions per block of 16 rows.)
template <int TYPE, int T, bool WHOLE>
__global__ void __launch_bounds__(SM_THREADS, 2) smallm_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ SmParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  using D = SmDec<TYPE>;
  constexpr bool PARTIAL = BlockTraits<TYPE>::QK == 32 && !WHOLE;   // a row may end inside a chunk
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + SM_MAX_STAGES;
  volatile int* s_last = reinterpret_cast<volatile int*>(empty + SM_MAX_STAGES);
  uint8_t* table = smem + 256;
  uint8_t* ring = table + sm_table_bytes<TYPE>();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], SM_WARPS);
    }
    fence_barrier_init();
  }
  if constexpr (sm_table_bytes<TYPE>() > 0) {
    const uint32_t* src = sm_table_source<TYPE>();
    for (int i = threadIdx.x; i < sm_table_bytes<TYPE>() / 4; i += SM_THREADS) reinterpret_cast<uint32_t*>(table)[i] = __ldg(src + i);
  }
  __syncthreads();
  const bool moe = p.passes != nullptr;
  const bool producer = warp == SM_WARPS;
  pdl_trigger();   // the next kernel may become resident; it waits for this one before it touches anything
  // The producer asks for weights first.  (Those of a MoE step too: the quantizer ahead let this kernel start when its own wait was
  // over, and the passes are older than that.  A step of eight tokens over 64 experts of Q4_0: 66.6 -> 61.6 us.)  The others wait when
  // they know their first tile.
  // units: chunk by chunk, row tile by row tile, pass by pass; CTA i owns the units [i * U / G, (i + 1) * U / G)
  // (the host sees to it that U * G fits 31 bits: everything here is 32-bit arithmetic, and divisions are few -- a 64-bit
  // division costs as much as a block of the product)
  const int n_passes = moe ? ld_older(p.n_passes) : 1;
  const int U = n_passes * p.rt * p.nc;
  const int G = U < (int)gridDim.x ? U : (int)gridDim.x;
  const int cta = (int)blockIdx.x;
  if (cta >= G) {
    pdl_wait();   // (not even a grid without work may complete before the kernels ahead of it)
    return;
  }
  const int u0 = (int)((unsigned)(cta * U) / (unsigned)G), u1 = (int)((unsigned)((cta + 1) * U) / (unsigned)G);
  const int first_tile = (int)((unsigned)u0 / (unsigned)p.nc);

  if (producer) {
    struct Cursor {   // a unit's row tile, chunk and (MoE) pass
      int c, r, pass;
      int4 info;      // {expert, first column tile, column tiles}
    };
    bool waited = false;
    auto load_pass = [&](Cursor& q) { q.info = !moe ? make_int4(0, 0, p.tiles, 0) : waited ? p.passes[q.pass] : ld_older(p.passes + q.pass); };
    auto advance = [&](Cursor& q) {
      if (++q.c == p.nc) {
        q.c = 0;
        if (++q.r == p.rt) { q.r = 0; ++q.pass; if (q.pass < n_passes) load_pass(q); }
      }
    };
    auto x_copy = [&](const Cursor& q, int s) {
      if (lane == 0)
        bulk_g2s(ring + (size_t)s * p.stage_bytes + p.raw.bytes, p.x + ((size_t)q.c * p.tiles + q.info.y) * SM_TILE_BYTES, (uint32_t)(q.info.z * SM_TILE_BYTES), &full[s]);
    };
    Cursor cur;
    cur.c = u0 - first_tile * p.nc;
    cur.pass = moe ? first_tile / p.rt : 0;
    cur.r = first_tile - cur.pass * p.rt;
    load_pass(cur);
    Cursor held = cur;        // first unit whose activations have not been asked for
    int n_held = 0, st = 0, st_in = 0;   // st_in: the stage that has to be there before the next one is asked for
    uint32_t ph = 0, ph_in = 0;
    auto release = [&]() {    // the activations exist now
      pdl_wait();
      waited = true;
      for (int v = 0; v < n_held; ++v) { x_copy(held, v); advance(held); }
    };
    for (int u = u0; u < u1; ++u) {
      if (!waited && n_held == p.ahead) release();
      if (u - u0 >= p.ahead) {
        if (!mbar_wait_bounded(&full[st_in], ph_in)) {
          if (lane == 0) atomicExch(p.status, E_TIMEOUT);
          drain_pause();
          break;
        }
        if (++st_in == p.stages) { st_in = 0; ph_in ^= 1u; }
      }
      if (!mbar_wait_bounded(&empty[st], ph ^ 1u)) {
        if (lane == 0) atomicExch(p.status, E_TIMEOUT);
        drain_pause();
        break;
      }
      raw_issue(p.raw, &map, p.w, p.w_bytes, cur.info.x * p.n, cur.r * RAW_ROWS, cur.c, ring + (size_t)st * p.stage_bytes, &full[st],
                (uint32_t)(cur.info.z * SM_TILE_BYTES), lane);
      __syncwarp();
      if (waited) x_copy(cur, st);
      else ++n_held;
      advance(cur);
      if (++st == p.stages) { st = 0; ph ^= 1u; }
    }
    if (!waited) release();
    return;
  }

  const int g = lane >> 2, t = lane & 3;
  const int r_lo = warp * 16 + g, r_hi = r_lo + 8;
  const uint32_t tab = smem_u32(table), ring_s = smem_u32(ring);
  int st = 0;
  uint32_t ph = 0;
  bool ok = true;
  constexpr int slot = SM_WARPS * 32 * T;   // float4s of a partial tile
  float4* part = reinterpret_cast<float4*>(p.part) + threadIdx.x;
  struct Shared { int n0, x0, nt, first, last, ta; };
  Shared shared_tile[2];                    // a contiguous range shares at most its first and its last tile
  int n_shared = 0;
  // Output rows of this lane's columns (rows_out and beyond: none) and their routing weights.  Asked for before a tile's
  // products, used behind them: two dependent loads from memory.
  struct Out { int row[T][2]; float scale[T][2]; };
  auto outputs = [&](Out& o, int x0, int nt) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = 8 * (x0 + i) + 2 * t + e;
        o.row[i][e] = i >= nt ? p.rows_out : moe ? __ldg(p.sorted + col) : (col < p.m ? col : p.rows_out);
        o.scale[i][e] = p.row_scale && o.row[i][e] < p.rows_out ? __ldg(p.row_scale + o.row[i][e]) : 1.f;
      }
    }
  };
  auto store = [&](const float (&acc)[T][4], int n0, const Out& o) {
#pragma unroll
    for (int i = 0; i < T; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = n0 + (e < 2 ? r_lo : r_hi), orow = o.row[i][e & 1];
        if (n < p.n && orow < p.rows_out) {
          switch (p.dtype) {
            case DT_F32: sm_store<float>(p, orow, n, acc[i][e], o.scale[i][e & 1]); break;
            case DT_F16: sm_store<__half>(p, orow, n, acc[i][e], o.scale[i][e & 1]); break;
            default: sm_store<__nv_bfloat16>(p, orow, n, acc[i][e], o.scale[i][e & 1]); break;
          }
        }
      }
    }
  };
  int u = u0, tile = first_tile, c0 = u0 - first_tile * p.nc;
  int pass = moe ? first_tile / p.rt : 0, r = first_tile - pass * p.rt;
  int4 pi = moe ? ld_older(p.passes + pass) : make_int4(0, 0, p.tiles, 0), pi_next = pi;
  pdl_wait();
  for (; u < u1; ++tile) {
    const int c1 = u1 - u < p.nc - c0 ? c0 + (u1 - u) : p.nc;
    const int nt = pi.z, x0 = pi.y, row0 = pi.x * p.n;
    if (moe && r + 1 == p.rt && u + (c1 - c0) < u1) pi_next = p.passes[pass + 1];   // (for the tile after this one)
    Out out_rows;
    constexpr bool early = T <= 2;   // (four column tiles have no registers left for it)
    if (early && c1 - c0 == p.nc) outputs(out_rows, x0, nt);
    const int n0 = r * RAW_ROWS;
    const uint32_t slot_lo = raw_slot(p.raw, r_lo, n0), slot_hi = raw_slot(p.raw, r_hi, n0);
    float acc[T][4];
#pragma unroll
    for (int i = 0; i < T; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int c = c0; c < c1; ++c) {
      if (ok && !mbar_wait_bounded(&full[st], ph)) {
        if (lane == 0) atomicExch(p.status, E_TIMEOUT);
        ok = false;   // keep the barrier protocol of the CTA going; the result is invalid and the status says so
      }
      const uint32_t base = sm_fresh(ring_s + (uint32_t)(st * p.stage_bytes));
      const uint32_t ra = base + slot_lo + (WHOLE ? 0u : raw_shift(p.raw, n0 + r_lo, row0, c));
      const uint32_t rb = base + slot_hi + (WHOLE ? 0u : raw_shift(p.raw, n0 + r_hi, row0, c));
      const uint32_t xt = base + (uint32_t)p.raw.bytes, xb = xt + 8u * lane, xd = xt + SM_CODE_BYTES + 16u * t;
      const int left = PARTIAL ? p.nblk - 8 * c : 8;
      if (ok) {
        typename D::Row ha, hb;
        D::head(ra, ha);
        D::head(rb, hb);
        if constexpr (D::MINS) {
          float la[2], ha2[2];
          const float fl = D::mins(ra, ha, t, left, la), fh = D::mins(rb, hb, t, left, ha2);
#pragma unroll
          for (int i = 0; i < T; ++i) {
            if (i == 0 || i < nt) {
              const uint4 s = sl128(xt + i * SM_TILE_BYTES + SM_CODE_BYTES + SM_PAIR_BYTES + 16u * lane);
              float c4[4] = {0.f, 0.f, 0.f, 0.f};
              sm_mma_tf32(c4, la, ha2, s.x, s.y);
              sm_mma_tf32(c4, la, ha2, s.z, s.w);
              acc[i][0] = fmaf(fl, c4[0], acc[i][0]);
              acc[i][1] = fmaf(fl, c4[1], acc[i][1]);
              acc[i][2] = fmaf(fh, c4[2], acc[i][2]);
              acc[i][3] = fmaf(fh, c4[3], acc[i][3]);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (!PARTIAL || j < left) {
            SmBlk lo, hi;
            if constexpr (sm_can_be_whole<TYPE>()) {
              D::template block<WHOLE>(ra, ha, j, t, tab, lo);
              D::template block<WHOLE>(rb, hb, j, t, tab, hi);
            } else {
              D::block(ra, ha, j, t, tab, lo);
              D::block(rb, hb, j, t, tab, hi);
            }
#pragma unroll
            for (int i = 0; i < T; ++i) {
              if (i == 0 || i < nt) {
                const uint2 b = sl64(xb + i * SM_TILE_BYTES + j * 256);
                const uint4 dq = sl128(xd + i * SM_TILE_BYTES + j * 64);
                sm_block<D::KIND, D::U8>(acc[i], lo, hi, b, make_float4(__uint_as_float(dq.x), __uint_as_float(dq.y), __uint_as_float(dq.z), __uint_as_float(dq.w)));
              }
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[st]);
      if (++st == p.stages) { st = 0; ph ^= 1u; }
    }
    // ---- the tile's sum: whole, or published for the last of the CTAs that share the tile ----
    if (c1 - c0 < p.nc) {
      // CTA q holds the units [q * U / G, (q + 1) * U / G): the ones that share this tile
      const int ta = tile * p.nc, k = n_shared++;
      Shared& sh = shared_tile[k];
      sh = {n0, x0, nt, (int)((unsigned)((ta + 1) * G - 1) / (unsigned)U), (int)((unsigned)((ta + p.nc) * G - 1) / (unsigned)U), ta};
      float4* out = part + (size_t)(2 * cta + (tile == first_tile ? 0 : 1)) * slot;
#pragma unroll
      for (int i = 0; i < T; ++i)
        if (i < nt) out[i * SM_WARPS * 32] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      asm volatile("bar.sync 1, %0;" ::"n"(SM_WARPS * 32) : "memory");
      if (threadIdx.x == 0) {   // (the other warps go on; the ring is deep enough to hide this one's wait)
        __threadfence();        // cumulative: covers what the barrier made visible to this thread
        s_last[k] = atomicAdd(p.counter + tile, 1) == sh.last - sh.first;
        __threadfence();
      }
    } else {
      if (!early) outputs(out_rows, x0, nt);
      store(acc, n0, out_rows);
    }
    u += c1 - c0;
    c0 = 0;
    if (++r == p.rt) { r = 0; ++pass; pi = pi_next; }
  }
  // The last CTA to arrive at a shared tile adds all its parts, in the order of the chunks: the same bits whoever it is.
  if (n_shared > 0) asm volatile("bar.sync 1, %0;" ::"n"(SM_WARPS * 32) : "memory");
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (k >= n_shared || s_last[k] == 0) continue;
    const Shared& sh = shared_tile[k];
    Out out_rows;
    outputs(out_rows, sh.x0, sh.nt);
    float acc[T][4];
#pragma unroll
    for (int i = 0; i < T; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    // (only the first of them can have come from an earlier tile, and keeps this one in its second slot)
    const int s_first = 2 * sh.first + ((unsigned)(sh.first * U) / (unsigned)G >= (unsigned)sh.ta ? 0 : 1);
    for (int q = sh.first; q <= sh.last; q += 8) {
#pragma unroll
      for (int i = 0; i < T; ++i) {
        if (i < sh.nt) {
          float4 v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            v[e] = q + e <= sh.last ? __ldcg(part + (size_t)(q + e == sh.first ? s_first : 2 * (q + e)) * slot + i * SM_WARPS * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            acc[i][0] += v[e].x; acc[i][1] += v[e].y; acc[i][2] += v[e].z; acc[i][3] += v[e].w;
          }
        }
      }
    }
    store(acc, sh.n0, out_rows);
  }
  if (!ok) drain_pause();   // copies in flight land before the CTA retires
}

template <int TYPE, int T, bool WHOLE> static int sm_launch_t(const SmParams& p, const CUtensorMap& map, int grid, size_t smem, cudaStream_t stream) {
  auto kern = smallm_kernel<TYPE, T, WHOLE>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess) return E_CUDA;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return E_CUDA;
    configured[dev & 63] = true;
  }
  return launch_pdl(kern, dim3((unsigned)grid), dim3(SM_THREADS), smem, stream, map, p) == cudaSuccess ? E_OK : E_CUDA;
}
template <int TYPE> int sm_launch(const SmParams& p, const CUtensorMap& map, int t, int grid, size_t smem, cudaStream_t stream) {
  if constexpr (sm_can_be_whole<TYPE>()) {
    if (p.raw.mode == 1 && p.nblk % 8 == 0) {
      switch (t) {
        case 1: return sm_launch_t<TYPE, 1, true>(p, map, grid, smem, stream);
        case 2: return sm_launch_t<TYPE, 2, true>(p, map, grid, smem, stream);
        case 4: return sm_launch_t<TYPE, 4, true>(p, map, grid, smem, stream);
      }
    }
  }
  switch (t) {
    case 1: return sm_launch_t<TYPE, 1, false>(p, map, grid, smem, stream);
    case 2: return sm_launch_t<TYPE, 2, false>(p, map, grid, smem, stream);
    case 4: return sm_launch_t<TYPE, 4, false>(p, map, grid, smem, stream);
  }
  return E_BAD_SHAPE;
}

}  // namespace gguf_b200
