// Instantiations of the shared-cache attention for one cache type.
#include "attn_mma.cuh"

namespace b200lm {
void launch_attn_shared_f32(cudaStream_t st, const AmArgs& a, int hd, int device, int sms, int cap, unsigned* tickets) {
  launch_attn_shared<float>(st, a, hd, device, sms, cap, tickets);
}
}  // namespace b200lm
