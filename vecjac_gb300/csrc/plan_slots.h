// Which slot of the batched SVD's plan memory a launch gets (host.cu): the numbers only, so that a host
// harness can run it. Callers hold a lock.
#pragma once
#include <vector>

namespace vj {
namespace host {

// Slots of launches that run when they are enqueued, in turn. A slot is held by the thread that
// enqueues until done(); a launch that gets a slot again is ordered behind the launch before by
// an event (`used`: there is one), so any number of them may be in flight on any streams.
struct EagerSlots {
  explicit EagerSlots(int n) : held((size_t)n, 0), used((size_t)n, 0) {}
  int take()
  {
    for (size_t k = 0; k < held.size(); ++k) {
      const int s = (int)(next++ % held.size());
      if (!held[(size_t)s]) {
        held[(size_t)s] = 1;
        return s;
      }
    }
    return -1;  // (as many threads as slots in the middle of a call)
  }
  void done(int s)
  {
    held[(size_t)s] = 0;
    used[(size_t)s] = 1;
  }
  std::vector<char> held, used;
  size_t next = 0;
};

// Slots of launches captured into a graph, which may run whenever the graph is replayed: a slot
// is its graph's until the graph and what was instantiated from it are gone (give_back).
struct GraphSlots {
  // a slot of no living graph; -1: all are taken, grow() first
  int take()
  {
    if (free_.empty())
      return -1;
    const int s = free_.back();
    free_.pop_back();
    return s;
  }
  void give_back(int s) { free_.push_back(s); }
  void grow(int n)
  {
    for (int k = n - 1; k >= 0; --k)
      free_.push_back(count + k);
    count += n;
  }
  int count = 0;

 private:
  std::vector<int> free_;
};

}  // namespace host
}  // namespace vj
