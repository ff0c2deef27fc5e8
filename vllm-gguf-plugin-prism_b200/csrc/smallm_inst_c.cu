// Instances of the small-batch kernel: code-book formats.
#include "smallm.cuh"

namespace gguf_b200 {
#define SM_INST(TYPE) template int sm_launch<TYPE>(const SmParams&, const CUtensorMap&, int, int, size_t, cudaStream_t);
SM_INST(T_IQ2_XXS)
SM_INST(T_IQ2_XS)
SM_INST(T_IQ2_S)
SM_INST(T_IQ3_XXS)
SM_INST(T_IQ3_S)
SM_INST(T_IQ1_S)
SM_INST(T_IQ1_M)
}  // namespace gguf_b200
