// Instances of the small-batch kernel: K formats.
#include "smallm.cuh"

namespace gguf_b200 {
#define SM_INST(TYPE) template int sm_launch<TYPE>(const SmParams&, const CUtensorMap&, int, int, size_t, cudaStream_t);
SM_INST(T_Q2_K)
SM_INST(T_Q3_K)
SM_INST(T_Q4_K)
SM_INST(T_Q5_K)
SM_INST(T_Q6_K)
}  // namespace gguf_b200
