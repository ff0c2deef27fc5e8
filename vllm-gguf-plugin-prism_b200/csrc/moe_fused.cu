// The small kernels that turn the MoE step around the two expert products into one call
// (reference: _fused_moe_gguf, quantization/fused_moe.py:56-133 -- there the alignment, the
// activation, the routing-weight multiply and the top-k sum are four separate library ops with
// their own launches and two [tokens*top_k, .] round trips through memory):
//
//   moe_plan_kernel    slots (token*top_k + j) sorted by expert, and the work list of the expert
//                      products.  Slots keep their order inside an expert (stable), so the result is unique.
//   moe_blocks_kernel  the work list for a caller's own block-aligned lists (ggml_moe_a8)
//   moe_sum_kernel     out[t] = sum over j of y[t*top_k + j]   (fp32 accumulation, one rounding)
//
// The activation (silu/gelu(gate) * up) runs inside the activation quantizer of the second product
// (quantize_q8_1.cu, act mode) and the routing weights inside that product's epilogue (mmq.cu, smallm.cu), so
// neither the activated matrix nor the weighted one exists in memory.
#include "common.cuh"
#include "kernels.h"

namespace gguf_b200 {

// One CTA.  Each of its 32 warps owns a contiguous run of slots and walks it twice, 32 slots at a time: first counting per
// expert (lanes with the same expert find one another with a match, their first lane adds), then placing, each slot at its
// expert's start + what earlier warps counted + what its own warp has placed so far.  (Three launches that scanned all slots
// once per expert took 28 us for 2048 slots and 64 experts; 512 slots and 64 experts with this form: see the MoE figures.)
constexpr int MOE_MAX_EXPERTS = 256;
__global__ void __launch_bounds__(1024) moe_plan_kernel(const int32_t* __restrict__ topk_ids, int slots, int n_experts, int align, int pass_rows,
                                                        int32_t* __restrict__ sorted, int4* __restrict__ passes, int32_t* __restrict__ n_passes) {
  pdl_trigger();
  __shared__ int32_t s_cnt[32][MOE_MAX_EXPERTS + 1];   // per warp and expert: counts, then the position of the warp's next slot
  __shared__ int32_t s_tot[MOE_MAX_EXPERTS], s_start[MOE_MAX_EXPERTS], s_pass[MOE_MAX_EXPERTS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = lane; e < n_experts; e += 32) s_cnt[warp][e] = 0;
  pdl_wait();
  __syncthreads();
  const int run = ((slots + 31) / 32 + 31) / 32 * 32, s0 = warp * run, s1 = min(slots, s0 + run), warps = (slots + run - 1) / run;   // warps that have slots
  for (int s = s0; s < s1; s += 32) {
    const int e = s + lane < s1 ? topk_ids[s + lane] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && e < n_experts && lane == __ffs(same) - 1) s_cnt[warp][e] += __popc(same);
    __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n_experts; e += blockDim.x) {   // per expert: prefix over the warps
    int c = 0;
    for (int w0 = 0; w0 < warps; w0 += 8) {   // (eight loads in flight)
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = s_cnt[w0 + i][e];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s_cnt[w0 + i][e] = c;
        c += v[i];
      }
    }
    s_tot[e] = c;
  }
  __syncthreads();
  if (warp == 0) {   // prefix sums over the experts: rows and passes
    int rows = 0, ps = 0;
    for (int e0 = 0; e0 < n_experts; e0 += 32) {
      const int e = e0 + lane, c = e < n_experts ? s_tot[e] : 0;
      const int nr = (c + align - 1) / align * align, np = (c + pass_rows - 1) / pass_rows;
      int a = nr, b = np;
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, a, m), v = __shfl_up_sync(0xffffffffu, b, m);
        if (lane >= m) { a += u; b += v; }
      }
      if (e < n_experts) {
        s_start[e] = rows + a - nr;
        s_pass[e] = ps + b - np;
      }
      rows += __shfl_sync(0xffffffffu, a, 31);
      ps += __shfl_sync(0xffffffffu, b, 31);
    }
    if (lane == 0) {
      n_passes[0] = ps;
      n_passes[1] = rows / align;
    }
  }
  __syncthreads();
  for (int e = warp; e < n_experts; e += 32) {
    const int c = s_tot[e], start = s_start[e];
    for (int i = lane; i < (c + pass_rows - 1) / pass_rows; i += 32) {
      const int left = c - i * pass_rows, n = left < pass_rows ? left : pass_rows;
      passes[s_pass[e] + i] = make_int4(e, (start + i * pass_rows) / align, (n + align - 1) / align, 0);
    }
    for (int i = start + c + lane; i < start + (c + align - 1) / align * align; i += 32) sorted[i] = slots;
  }
  for (int s = s0; s < s1; s += 32) {
    const int e = s + lane < s1 ? topk_ids[s + lane] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const bool valid = e >= 0 && e < n_experts;
    const int at = valid ? s_start[e] + s_cnt[warp][e] + __popc(same & ((1u << lane) - 1u)) : 0;
    __syncwarp();
    if (valid) {
      sorted[at] = s + lane;
      if (lane == __ffs(same) - 1) s_cnt[warp][e] += __popc(same);
    }
    __syncwarp();
  }
}

int64_t moe_plan_rows(int64_t slots, int n_experts, int align) {
  const int64_t worst = slots + (int64_t)n_experts * (align - 1);      // every expert may leave part of a group unfilled
  return (slots * align < worst ? slots * align : worst) / align * align;
}
int64_t moe_plan_passes(int64_t slots, int n_experts, int pass_rows) {
  const int64_t worst = slots / pass_rows + n_experts;
  return slots < worst ? slots : worst;
}
int launch_moe_plan(const int32_t* topk_ids, int64_t slots, int n_experts, int align, int pass_rows, int32_t* sorted, void* passes,
                    int32_t* n_passes, cudaStream_t stream) {
  if (n_experts < 1 || n_experts > MOE_MAX_EXPERTS || slots > 1 << 24) return E_BAD_SHAPE;
  return launch_pdl(moe_plan_kernel, dim3(1), dim3(1024), 0, stream, topk_ids, (int)slots, n_experts, align, pass_rows, sorted,
                    static_cast<int4*>(passes), n_passes) == cudaSuccess ? E_OK : E_CUDA;
}

__global__ void __launch_bounds__(1024) moe_blocks_kernel(const int32_t* __restrict__ expert_ids, const int32_t* __restrict__ n_post_pad, int n_sorted,
                                                          int n_experts, int block, int4* __restrict__ passes, int32_t* __restrict__ n_passes) {
  pdl_trigger();
  pdl_wait();
  __shared__ int32_t s_base, s_warp[32];
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  const int rows = min(n_post_pad[0], n_sorted), blocks = (rows + block - 1) / block;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b0 = 0; b0 < blocks; b0 += blockDim.x) {
    const int b = b0 + threadIdx.x;
    const int e = b < blocks ? expert_ids[b] : -1;
    const bool use = e >= 0 && e < n_experts;
    const unsigned m = __ballot_sync(0xffffffffu, use);
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int at = s_base + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) at += s_warp[w];
    if (use) passes[at] = make_int4(e, b * block, min(block, rows - b * block), 0);
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < 32; ++w) s_base += s_warp[w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    n_passes[0] = s_base;
    n_passes[1] = rows;
  }
}
int launch_moe_blocks(const int32_t* expert_ids, const int32_t* n_post_pad, int64_t n_sorted, int n_experts, int block, void* passes,
                      int32_t* n_passes, cudaStream_t stream) {
  return launch_pdl(moe_blocks_kernel, dim3(1), dim3(1024), 0, stream, expert_ids, n_post_pad, (int)n_sorted, n_experts, block,
                    static_cast<int4*>(passes), n_passes) == cudaSuccess ? E_OK : E_CUDA;
}

// Eight columns per thread.  (One column per thread, with a 64-bit division for it, took 10.4 us for 256 tokens of 2048
// columns and eight experts, 278 instructions a column; the traffic is worth 1.5 us.)
template <typename T>
__global__ void __launch_bounds__(256) moe_sum_kernel(const T* __restrict__ y, T* __restrict__ out, const int32_t* __restrict__ topk_ids,
                                                      int n_experts, int64_t tokens, int top_k, int64_t h) {
  pdl_trigger();
  pdl_wait();
  constexpr int W = sizeof(T) / 2;               // 16-byte words of eight values
  const unsigned per_row = (unsigned)(h / 8);
  const int64_t total = tokens * per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned t = (unsigned)i / per_row;
    const int64_t c = 8 * (int64_t)((unsigned)i - t * per_row);
    const int32_t* ids = topk_ids + (int64_t)t * top_k;
    const T* in = y + (int64_t)t * top_k * h + c;
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = 0.f;
#pragma unroll 4
    for (int j = 0; j < top_k; ++j, in += h) {
      const int e = __ldg(ids + j);
      if (e < 0 || e >= n_experts) continue;     // a slot without a valid expert contributes nothing
      uint4 v[W];
#pragma unroll
      for (int k = 0; k < W; ++k) v[k] = reinterpret_cast<const uint4*>(in)[k];
#pragma unroll
      for (int k = 0; k < 8; ++k) s[k] += to_float<T>(reinterpret_cast<const T*>(v)[k]);
    }
    uint4 o[W];
#pragma unroll
    for (int k = 0; k < 8; ++k) reinterpret_cast<T*>(o)[k] = from_float<T>(s[k]);
#pragma unroll
    for (int k = 0; k < W; ++k) reinterpret_cast<uint4*>(out + (int64_t)t * h + c)[k] = o[k];
  }
}

int launch_moe_sum(const void* y, void* out, const int32_t* topk_ids, int n_experts, int64_t tokens, int64_t top_k, int64_t h,
                   int dtype, cudaStream_t stream) {
  if (h % 8 != 0) return E_BAD_SHAPE;
  const int64_t total = tokens * (h / 8);
  if (total == 0) return E_OK;
  if (total >= (int64_t)1 << 32) return E_TOO_LARGE;
  const unsigned grid = (unsigned)((total + 255) / 256 > 148 * 8 ? 148 * 8 : (total + 255) / 256);
  cudaError_t e;
  switch (dtype) {
    case DT_F32:
      e = launch_pdl(moe_sum_kernel<float>, dim3(grid), dim3(256), 0, stream, (const float*)y, (float*)out, topk_ids, n_experts, tokens, (int)top_k, h);
      break;
    case DT_F16:
      e = launch_pdl(moe_sum_kernel<__half>, dim3(grid), dim3(256), 0, stream, (const __half*)y, (__half*)out, topk_ids, n_experts, tokens, (int)top_k, h);
      break;
    case DT_BF16:
      e = launch_pdl(moe_sum_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, stream, (const __nv_bfloat16*)y, (__nv_bfloat16*)out, topk_ids, n_experts, tokens, (int)top_k, h);
      break;
    default:
      return E_BAD_DTYPE;
  }
  return e == cudaSuccess ? E_OK : E_CUDA;
}

}  // namespace gguf_b200
