// Instances of the tensor-core GEMM: IQ1 and IQ4 formats.
#include "mmq_kernel.cuh"

namespace gguf_b200 {
#define MMQ_INST(TYPE) template int mmq_launch<TYPE>(const MmqParams&, const CUtensorMap&, const CUtensorMap&, int, bool, int, size_t, cudaStream_t);
MMQ_INST(T_IQ1_S)
MMQ_INST(T_IQ1_M)
MMQ_INST(T_IQ4_NL)
MMQ_INST(T_IQ4_XS)
}  // namespace gguf_b200
