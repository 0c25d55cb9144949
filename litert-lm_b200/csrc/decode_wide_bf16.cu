// Instantiations of the wide decode step's attention for one cache type.
#include "decode_wide.cuh"

namespace b200lm {
void launch_wide_attn_bf16(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a) {
  launch_wide_attn_h<__nv_bfloat16>(st, d, nb, smem_optin, a);
}
}  // namespace b200lm
