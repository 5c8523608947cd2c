// What has to be done once for every device of a process (a kernel's permissions are a device's own).
#pragma once
#include <atomic>
#include <cstdint>

namespace us {

class OncePerDevice {
 public:
  // f() unless it has returned 0 for `device` before; its result, else 0.  Devices past 64 do it each time.
  template <typename F>
  int operator()(int device, F f) {
    const uint64_t bit = device < 64 ? 1ull << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = f();
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace us
