// Instances of the tensor-core GEMM: 32-value block formats.
#include "mmq_kernel.cuh"

namespace gguf_b200 {
#define MMQ_INST(TYPE) template int mmq_launch<TYPE>(const MmqParams&, const CUtensorMap&, const CUtensorMap&, int, bool, int, size_t, cudaStream_t);
MMQ_INST(T_Q4_0)
MMQ_INST(T_Q4_1)
MMQ_INST(T_Q5_0)
MMQ_INST(T_Q5_1)
MMQ_INST(T_Q8_0)
}  // namespace gguf_b200
