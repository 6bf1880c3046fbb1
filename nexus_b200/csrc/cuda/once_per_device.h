// Work that a process does once per device, such as allowing a kernel more dynamic shared memory than the default: an attribute of a
// function holds for the device that was current when it was set.
#pragma once
#include <atomic>
#include <cstdint>

namespace nx {

// Runs `work(device)` (0 = success) unless it has succeeded for this device before; 64 devices are remembered.  Threads that meet here
// may both run it.
class OncePerDevice {
 public:
  template <typename F>
  int operator()(int device, F work) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = work(device);
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace nx
