// Host side of the weight streaming (raw_stream.cuh): which form a matrix takes, and its tensor map.
#include "raw_stream.cuh"

namespace gguf_b200 {

EncodeTiledFn tensor_map_encoder() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
               ? reinterpret_cast<EncodeTiledFn>(p)
               : nullptr;
  }();
  return fn;
}

// (a row that ends between two words could only be described together with what follows it)
bool raw_dense(int type, int64_t K, int64_t pitch) {
  const int qk = block_size(type), ts = type_size(type);
  return RAW_KC / qk * ts % 16 == 0 && pitch % 16 == 0 && K / qk * ts % 4 == 0;
}

bool plan_raw(int type, const void* w, int64_t n_rows, int64_t copies, int64_t K, int64_t pitch, RawPlan& p, CUtensorMap& map, int64_t gap) {
  const int qk = block_size(type), ts = type_size(type);
  p = RawPlan{};
  p.pitch = pitch;
  p.row_bytes = K / qk * ts;
  p.rbc = RAW_KC / qk * ts;
  p.gap = copies > 1 ? gap : 0;
  p.nrows = p.nfull = (int)n_rows;
  if (pitch % raw_type_align(type) != 0 || pitch < p.row_bytes) return false;
  const int s16 = (p.rbc + 30) / 16;   // the chunk, displaced by up to 15 bytes
  p.slot = (s16 % 2 ? s16 : s16 + 1) * 16;
  EncodeTiledFn enc = tensor_map_encoder();
  auto encode = [&](int64_t inner, int64_t row, int64_t rows, int box0, int box1) {
    const cuuint32_t estr[2] = {1, 1};
    const cuuint64_t wd[2] = {(cuuint64_t)(inner / 4), (cuuint64_t)rows};
    const cuuint64_t ws[1] = {(cuuint64_t)row};
    const cuuint32_t wb[2] = {(cuuint32_t)(box0 / 4), (cuuint32_t)box1};
    return enc && enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(w), wd, ws, wb, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (p.gap != 0) {
    // rows of such matrices have no common distance: one copy each
  } else if (const int odd = p.rbc | 16; raw_dense(type, K, pitch) && encode(p.row_bytes, pitch, n_rows * copies, odd, RAW_ROWS)) {
    p.mode = 1;
    p.slot = odd;   // (behind a chunk of an even number of units, the start of the next: Q4_1 14336x4096, 48 tokens 26.5 -> 21.7 us, Q5_1 31.5 -> 24.2)
  } else {
    int cl = 0;
    while (((pitch << cl) & 15) != 0) ++cl;
    const int64_t covered = n_rows >> cl << cl;
    if (covered > 0 && (covered == n_rows || copies == 1) && encode(pitch << cl, pitch << cl, (covered >> cl) * copies, p.slot, RAW_ROWS >> cl)) {
      p.mode = 2;
      p.cl2 = cl;
      p.nfull = (int)covered;
    }
  }
  p.bytes = (int)round_up((int64_t)(RAW_ROWS + (p.nfull < p.nrows ? RAW_EXTRA : 0)) * p.slot, 128);
  return true;
}

}  // namespace gguf_b200
