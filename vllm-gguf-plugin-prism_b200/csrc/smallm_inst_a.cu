// Instances of the small-batch kernel: 32-value block formats.
#include "smallm.cuh"

namespace gguf_b200 {
#define SM_INST(TYPE) template int sm_launch<TYPE>(const SmParams&, const CUtensorMap&, int, int, size_t, cudaStream_t);
SM_INST(T_Q4_0)
SM_INST(T_Q4_1)
SM_INST(T_Q5_0)
SM_INST(T_Q5_1)
SM_INST(T_Q8_0)
SM_INST(T_IQ4_NL)
SM_INST(T_IQ4_XS)
}  // namespace gguf_b200
