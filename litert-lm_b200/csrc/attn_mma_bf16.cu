// Instantiations of the shared-cache attention for one cache type.
#include "attn_mma.cuh"

namespace b200lm {
void launch_attn_shared_bf16(cudaStream_t st, const AmArgs& a, int hd, int device, int sms, int cap, unsigned* tickets) {
  launch_attn_shared<__nv_bfloat16>(st, a, hd, device, sms, cap, tickets);
}
}  // namespace b200lm
