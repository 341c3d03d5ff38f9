// Host harness for the slots of the batched SVD's plan memory (vecjac_gb300/csrc/plan_slots.h):
// prints "ok" or the first violation.
#include <cstdio>
#include <set>
#include <vector>

#include "../vecjac_gb300/csrc/plan_slots.h"

static int fail(const char *what)
{
  std::printf("%s\n", what);
  return 1;
}

int main()
{
  using namespace vj::host;
  // eager: no slot twice while it is held; a slot that comes again is marked as used
  EagerSlots e(8);
  std::set<int> held;
  for (int k = 0; k < 8; ++k) {
    const int s = e.take();
    if (s < 0 || s >= 8 || !held.insert(s).second)
      return fail("a held slot was handed out");
    if (e.used[(size_t)s])
      return fail("a fresh slot is marked as used");
  }
  if (e.take() != -1)
    return fail("a ninth slot of eight");
  e.done(5);
  if (e.take() != 5 || !e.used[5])
    return fail("the one free slot, used before");
  for (int s = 0; s < 8; ++s)
    e.done(s);
  int last = -1;
  for (int k = 0; k < 100; ++k) {
    const int s = e.take();
    if (s == last)
      return fail("slots do not take turns");
    e.done(s);
    last = s;
  }
  // graphs: thousands of captured launches among eager ones share no slot while their graphs live
  GraphSlots g;
  std::set<int> live;
  std::vector<int> order;
  for (int k = 0; k < 5000; ++k) {
    int s = g.take();
    if (s < 0) {
      g.grow(64);
      s = g.take();
    }
    if (s < 0 || s >= g.count || !live.insert(s).second)
      return fail("a living graph's slot was handed out");
    order.push_back(s);
    if (k % 3 == 2) {
      const int r = order[(size_t)(k / 3)];
      live.erase(r);
      g.give_back(r);
    }
  }
  if (g.count > (int)live.size() + 1 + 64)
    return fail("slots are not reused");
  std::printf("ok\n");
  return 0;
}
