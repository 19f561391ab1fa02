// Shares the device's SMs among the nodal phases of concurrent solves: of
// usap_batch_partition, of servers and of contexts on several threads.  Each
// phase is one cooperative launch of as many CTAs (one per SM) as it is given
// here, so the phases of different solves run side by side on disjoint SMs,
// and a solve's merge phase and host steps overlap the others' phases.
//
// A phase's CTAs wait for one another, so all of them have to be resident
// while it runs: a launch whose CTAs partly queue behind another phase would
// spin until that phase ends, or until its barrier gives up.  One pool per
// device therefore hands out the CTAs of every phase of the process, never
// more than are resident together.
//
// A phase's share follows its batch size among the solves in progress, so
// that large and small graphs advance at about the same rate, up to a warp
// per batch vertex (more CTAs would idle).  Fewer CTAs per solve are more
// efficient: a batch has a fixed cost per CTA (two grid barriers, a chain of
// dependent loads per proposal) of about 12 us.  Phases are admitted in
// arrival order, and may start on half their share when no more is free.  A
// context's solve takes every SM while it is alone: its latency counts, and
// the warps beyond one per vertex help with the float dS.
// The merge phases' ordinary kernels run on what is free; keeping SMs out of
// the pool for them was slower (12 graphs x 4 chains: 594 ms without, 625 ms
// with 12 kept free).
#include "smpool.h"

#include <algorithm>
#include <map>

namespace usap {

std::shared_ptr<SmPool> SmPool::of_device(int device, int total, int warps) {
  static std::mutex mu;
  static std::map<int, std::weak_ptr<SmPool>> pools;
  std::lock_guard<std::mutex> lk(mu);
  std::shared_ptr<SmPool> p = pools[device].lock();
  if (!p) pools[device] = p = std::make_shared<SmPool>(total, warps);
  return p;
}

void SmPool::enter(int64_t batch) {
  std::lock_guard<std::mutex> lk(mu_);
  solves_++;
  live_ += batch;
}

void SmPool::leave(int64_t batch) {
  std::lock_guard<std::mutex> lk(mu_);
  solves_--;
  live_ -= batch;
}

bool SmPool::shared() {
  std::lock_guard<std::mutex> lk(mu_);
  return solves_ > 1;
}

int SmPool::acquire(int64_t batch, int most, bool whole) {
  std::unique_lock<std::mutex> lk(mu_);
  const uint64_t ticket = next_++;
  cv_.wait(lk, [&] { return ticket == serving_; });
  most = std::min(most, total_);
  int want = most;
  if (!whole || solves_ > 1) {
    const int64_t useful = std::min<int64_t>((batch + warps_ - 1) / warps_, most);
    const int64_t share = total_ * batch / std::max<int64_t>(live_, batch);
    want = static_cast<int>(std::max<int64_t>(1, std::min(share, useful)));
  }
  cv_.wait(lk, [&] { return 2 * free_ >= want; });
  const int got = std::max(1, std::min(want, free_));
  free_ -= got;
  serving_++;
  lk.unlock();
  cv_.notify_all();
  return got;
}

void SmPool::release(int ctas) {
  {
    std::lock_guard<std::mutex> lk(mu_);
    free_ += ctas;
  }
  cv_.notify_all();
}

}  // namespace usap
