// Set-up that has to be done once on every device of the process (a kernel's
// shared-memory opt-in applies to the current device only).
#pragma once
#include <atomic>

namespace bem {

class OncePerDevice {
 public:
  // configure() on the first call for the device and again until it returns 0
  // (its status is returned).  Any number of threads: two that come first
  // together both run it, so it must be harmless to repeat.  A device index
  // beyond the table is configured on every call.
  template <class Configure>
  int operator()(int device, Configure&& configure) {
    const bool known = device >= 0 && device < kDevices;
    if (known && done_[device].load(std::memory_order_acquire)) return 0;
    const int status = configure();
    if (status == 0 && known) done_[device].store(true, std::memory_order_release);
    return status;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace bem
