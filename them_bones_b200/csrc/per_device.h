// Host code that has to run once on each device of a process: a kernel's shared-memory limit, for one, belongs to the device that is
// current when it is set, and a launch on another device that asks for more than 48 KB fails without it.
#pragma once
#include <atomic>

namespace bones {

class OncePerDevice {
 public:
  static constexpr int kDevices = 64;
  // Runs `set` (0 or an error code) unless it has succeeded on device `dev` before.  After an error, and on devices past the table, it
  // runs again; two threads that come at the same time may both run it.
  template <class Set>
  int operator()(int dev, Set set) {
    const bool kept = dev >= 0 && dev < kDevices;
    if (kept && done_[dev].load(std::memory_order_acquire)) return 0;
    const int rc = set();
    if (rc == 0 && kept) done_[dev].store(true, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace bones
