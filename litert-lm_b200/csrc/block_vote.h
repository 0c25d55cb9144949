// How the threads of a block part where a bounded wait may have given up.  Not every thread's wait does, and a word that all
// of them read can change while they read it: one that saw the sign and one that did not would go on to different barriers
// and wait there for each other.  So every thread brings what it knows to the barrier and takes the barrier's answer, which
// is the same for all: whether anyone had seen it.  A sign that appears later is the next vote's.
#pragma once

#ifdef __CUDACC__
#define B2_VOTE_FN __host__ __device__ __forceinline__
#else
#define B2_VOTE_FN inline
#endif

namespace b200lm {

// `seen` is this thread's look; `vote` is a barrier of all threads concerned that returns the or of what they bring.
template <typename Seen, typename Vote>
B2_VOTE_FN bool block_gave_up(const Seen& seen, const Vote& vote) {
  const bool mine = seen();
  return vote(mine);
}

}  // namespace b200lm
