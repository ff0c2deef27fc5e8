// Instances of the tensor-core GEMM: IQ2 and IQ3 formats.
#include "mmq_kernel.cuh"

namespace gguf_b200 {
#define MMQ_INST(TYPE) template int mmq_launch<TYPE>(const MmqParams&, const CUtensorMap&, const CUtensorMap&, int, bool, int, size_t, cudaStream_t);
MMQ_INST(T_IQ2_XXS)
MMQ_INST(T_IQ2_XS)
MMQ_INST(T_IQ2_S)
MMQ_INST(T_IQ3_XXS)
MMQ_INST(T_IQ3_S)
}  // namespace gguf_b200
