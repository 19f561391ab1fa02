// Accounting of SmPool with users of every kind on threads: contexts (the
// whole device while alone), batches and servers.  Prints "ok" or what failed.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "smpool.h"

using usap::SmPool;

namespace {
constexpr int kTotal = 148, kWarps = 24;
std::atomic<int> held{0}, failures{0};

void fail(const char* what) {
  std::printf("%s\n", what);
  failures++;
}

// one solve of `phases` nodal phases
void solve(int64_t batch, int most, bool whole, int phases) {
  std::shared_ptr<SmPool> p = SmPool::of_device(0, kTotal, kWarps);   // as every solver state does
  p->enter(batch);
  for (int k = 0; k < phases; k++) {
    const int n = p->acquire(batch, most, whole);
    const int now = held += n;
    if (n < 1 || n > most) fail("a share outside 1..most");
    if (now > kTotal) fail("more CTAs given out than are resident");
    std::this_thread::yield();
    held -= n;
    p->release(n);
  }
  p->leave(batch);
}
}  // namespace

int main() {
  {
    auto a = SmPool::of_device(0, kTotal, kWarps), b = SmPool::of_device(0, kTotal, kWarps);
    if (a != b) fail("two users of one device have two pools");
    if (a == SmPool::of_device(1, kTotal, kWarps)) fail("two devices share a pool");
    // alone, a context's solve gets what it asks for, whatever its batch size
    a->enter(100);
    if (a->shared()) fail("alone, but shared");
    for (int most : {kTotal, 8, 1, 2 * kTotal}) {
      const int n = a->acquire(100, most, true);
      if (n != (most < kTotal ? most : kTotal)) fail("a lone context's solve does not get all it may use");
      a->release(n);
    }
    // a batch's job gets a warp per batch vertex
    int n = a->acquire(100, kTotal, false);
    if (n != 5) fail("a lone job's share is not a warp per vertex");
    // beside it, a context's solve fits in what is left
    b->enter(100000);
    if (!a->shared()) fail("two solves, not shared");
    int m = b->acquire(100000, kTotal, true);
    if (n + m > kTotal) fail("two phases do not fit together");
    b->release(m);
    a->release(n);
    a->leave(100);
    b->leave(100000);
  }
  std::vector<std::thread> th;
  for (int i = 0; i < 12; i++)
    th.emplace_back([i] { solve(100ll << i, i % 5 == 4 ? 1 + i : kTotal, i % 3 == 0, 400); });
  for (auto& t : th) t.join();
  if (held != 0) fail("CTAs not given back");
  // everything was given back: a lone solve has the device again
  auto p = SmPool::of_device(0, kTotal, kWarps);
  p->enter(1);
  const int n = p->acquire(1, kTotal, true);
  if (n != kTotal) fail("CTAs lost");
  p->release(n);
  p->leave(1);
  if (!failures) std::printf("ok\n");
  return failures ? 1 : 0;
}
