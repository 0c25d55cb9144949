// Instantiations of the streaming decode kernel for one cache type.
#include "decode_stream.cuh"

namespace b200lm {
const void* decode_stream_kernel_bf16(const ModelDims& d) { return decode_stream_kernel_pick<__nv_bfloat16>(d); }
}  // namespace b200lm
