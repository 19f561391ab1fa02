// Shares the device's SMs among the nodal phases of concurrent solves
// (usap_batch_partition, the served form).  Each phase is one cooperative
// launch of as many CTAs (one per SM) as it is given here, so the phases of
// different solves run side by side on disjoint SMs, and a solve's merge
// phase and host steps overlap the others' phases.
//
// A phase's share follows its batch size among the solves in progress, so
// that large and small graphs advance at about the same rate, up to a warp
// per batch vertex (more CTAs would idle).  Fewer CTAs per solve are more
// efficient: a batch has a fixed cost per CTA (two grid barriers, a chain of
// dependent loads per proposal) of about 12 us.  Phases are admitted in
// arrival order, and may start on half their share when no more is free.
// The merge phases' ordinary kernels run on what is free; keeping SMs out of
// the pool for them was slower (12 graphs x 4 chains: 594 ms without, 625 ms
// with 12 kept free).
#include <algorithm>

#include "job.h"

namespace usap {

SmPool::SmPool(int device) { total_ = free_ = nodal_phase_grid(device); }

void SmPool::enter(int64_t batch) {
  std::lock_guard<std::mutex> lk(mu_);
  live_ += batch;
}

void SmPool::leave(int64_t batch) {
  std::lock_guard<std::mutex> lk(mu_);
  live_ -= batch;
}

int SmPool::acquire(int64_t batch, int most) {
  std::unique_lock<std::mutex> lk(mu_);
  const uint64_t ticket = next_++;
  cv_.wait(lk, [&] { return ticket == serving_; });
  const int64_t warps = nodal_phase_warps();
  const int64_t useful = std::min<int64_t>((batch + warps - 1) / warps, std::min(most, total_));
  const int64_t share = total_ * batch / std::max<int64_t>(live_, batch);
  const int want = static_cast<int>(std::max<int64_t>(1, std::min(share, useful)));
  cv_.wait(lk, [&] { return 2 * free_ >= want; });
  const int got = std::max(1, std::min(want, free_));
  free_ -= got;
  serving_++;
  launches_++;
  lk.unlock();
  cv_.notify_all();
  return got;
}

void SmPool::release(int ctas, double ms) {
  {
    std::lock_guard<std::mutex> lk(mu_);
    free_ += ctas;
    ms_ += ms;
  }
  cv_.notify_all();
}

}  // namespace usap
