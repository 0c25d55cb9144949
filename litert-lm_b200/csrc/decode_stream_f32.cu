// Instantiations of the streaming decode kernel for one cache type.
#include "decode_stream.cuh"

namespace b200lm {
const void* decode_stream_kernel_f32(const ModelDims& d) { return decode_stream_kernel_pick<float>(d); }
}  // namespace b200lm
