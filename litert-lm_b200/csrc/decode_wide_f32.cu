// Instantiations of the wide decode step's attention for one cache type.
#include "decode_wide.cuh"

namespace b200lm {
void launch_wide_attn_f32(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a) {
  launch_wide_attn_h<float>(st, d, nb, smem_optin, a);
}
}  // namespace b200lm
