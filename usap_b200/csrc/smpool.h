// The SMs of a device, shared by the nodal phases of the process's solves
// (smpool.cpp).
#pragma once

#include <condition_variable>
#include <cstdint>
#include <memory>
#include <mutex>

namespace usap {

class SmPool {
 public:
  // the device's pool: one for all contexts, batches and servers of the
  // process, kept while any of them holds it.  total: CTAs that are resident
  // together; warps: of each
  static std::shared_ptr<SmPool> of_device(int device, int total, int warps);
  SmPool(int total, int warps) : total_(total), free_(total), warps_(warps) {}
  SmPool(const SmPool&) = delete;
  SmPool& operator=(const SmPool&) = delete;
  // a solve with batches of `batch` vertices starts / ends
  void enter(int64_t batch);
  void leave(int64_t batch);
  // CTAs for its next nodal phase, at most `most` (waits for them), given back
  // when the phase is over.  whole: all `most` while it is the only solve
  int acquire(int64_t batch, int most, bool whole);
  void release(int ctas);
  // other solves are in progress beside the caller's
  bool shared();

 private:
  std::mutex mu_;
  std::condition_variable cv_;
  const int total_;
  int free_;
  const int warps_;
  int solves_ = 0;
  int64_t live_ = 0;                  // batch vertices of the solves in progress
  uint64_t next_ = 0, serving_ = 0;   // phases are admitted in arrival order
};

}  // namespace usap
