// Instantiations of the chained decode kernel for one cache type.
#include "decode_fused.cuh"

namespace b200lm {
const void* decode_fused_kernel_f32(const ModelDims& d) { return decode_fused_kernel_pick<float>(d); }
}  // namespace b200lm
