// Instances of the tensor-core GEMM: K formats.
#include "mmq_kernel.cuh"

namespace gguf_b200 {
#define MMQ_INST(TYPE) template int mmq_launch<TYPE>(const MmqParams&, const CUtensorMap&, const CUtensorMap&, int, bool, int, size_t, cudaStream_t);
MMQ_INST(T_Q2_K)
MMQ_INST(T_Q3_K)
MMQ_INST(T_Q4_K)
MMQ_INST(T_Q5_K)
MMQ_INST(T_Q6_K)
}  // namespace gguf_b200
