// Threads of a block that look for the sign of a wait that gave up, in every combination of who sees it when: all must go
// on the same way, and together, or some of them would wait at a barrier that the others never come to.
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

#include "block_vote.h"

using namespace b200lm;

// A block's barrier with an or over what the threads bring (__syncthreads_or).  A thread that waits for a minute says so.
class Barrier {
 public:
  explicit Barrier(int n) : n_(n) {}
  bool operator()(bool x) {
    std::unique_lock<std::mutex> lock(mu_);
    const long turn = turn_;
    any_ = any_ || x;
    if (++here_ == n_) {
      answer_ = any_;
      any_ = false;
      here_ = 0;
      ++turn_;
      cv_.notify_all();
      return answer_;
    }
    if (!cv_.wait_for(lock, std::chrono::seconds(60), [&] { return turn_ != turn; })) stuck = true;
    return answer_;
  }
  bool stuck = false;

 private:
  const int n_;
  int here_ = 0;
  long turn_ = 0;
  bool any_ = false, answer_ = false;
  std::mutex mu_;
  std::condition_variable cv_;
};

constexpr int kThreads = 4, kRounds = 3;

// first[i]: the round in which thread i sees the sign for the first time (kRounds: in none).  Returns the round each leaves in.
static std::vector<int> leave(const std::vector<int>& first, bool* stuck) {
  Barrier barrier(kThreads);
  std::vector<int> out(kThreads, kRounds);
  std::vector<std::thread> ts;
  for (int i = 0; i < kThreads; ++i)
    ts.emplace_back([&, i] {
      for (int r = 0; r < kRounds; ++r)
        if (block_gave_up([&] { return r >= first[i]; }, [&](bool x) { return barrier(x); })) { out[i] = r; break; }
    });
  for (std::thread& t : ts) t.join();
  *stuck = barrier.stuck;
  return out;
}

int main() {
  int combos = 1;
  for (int i = 0; i < kThreads; ++i) combos *= kRounds + 1;
  for (int c = 0; c < combos; ++c) {
    std::vector<int> first(kThreads);
    int least = kRounds;
    for (int i = 0, x = c; i < kThreads; ++i, x /= kRounds + 1) {
      first[i] = x % (kRounds + 1);
      least = first[i] < least ? first[i] : least;
    }
    bool stuck = false;
    for (int r : leave(first, &stuck))
      if (r != least || stuck) {
        printf("seen in rounds %d %d %d %d: a thread left in %d\n", first[0], first[1], first[2], first[3], r);
        return 1;
      }
  }
  printf("ok\n");
  return 0;
}
