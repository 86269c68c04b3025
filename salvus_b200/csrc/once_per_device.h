// once_per_device.h -- one-time set-up that belongs to a device.
#pragma once

#include <atomic>
#include <cstdint>

namespace salvus {

// Runs `set` (0: done) the first time a device needs it, and again after a
// failure: a kernel's attributes belong to the device that is current when they
// are set, not to the process.  Problems are prepared on several threads; two
// that arrive together both run `set`, which must bear that.  Devices from 64 on
// set every time.
class OncePerDevice {
 public:
  template <class F>
  int operator()(int device, F set) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = set();
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace salvus
