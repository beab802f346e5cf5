// The dynamic shared memory that a kernel may be launched with, raised as launches ask for more and never lowered.
//
// One object per kernel (a static of the function that launches it).  Launches of one kernel come from several threads with
// different sizes: a limit set to a call's own size could be lowered between another thread's request and its launch, which
// then fails.  `set(bytes)` sets the kernel's limit on the current device and returns 0, or an error code that is passed on.
#pragma once
#include <cstddef>
#include <mutex>

namespace tlx {

class SmemLimit {
 public:
  template <typename Set>
  int raise(int device, size_t bytes, Set&& set) {
    if (bytes <= kDefault) return 0;
    std::lock_guard<std::mutex> lock(mu_);
    const bool known = device >= 0 && device < kDevices;
    size_t& limit = limit_[known ? device : kDevices];   // (the last one: the greatest of all other devices, set every time)
    if (known && limit >= bytes) return 0;
    const size_t want = limit > bytes ? limit : bytes;
    const int rc = set(want);
    if (rc == 0) limit = want;
    return rc;
  }

 private:
  static constexpr size_t kDefault = 48 * 1024;   // what every kernel may use as it is
  static constexpr int kDevices = 64;
  std::mutex mu_;
  size_t limit_[kDevices + 1] = {};
};

}  // namespace tlx
