// Instantiations of the chained decode kernel for one cache type.
#include "decode_fused.cuh"

namespace b200lm {
const void* decode_fused_kernel_bf16(const ModelDims& d) { return decode_fused_kernel_pick<__nv_bfloat16>(d); }
}  // namespace b200lm
