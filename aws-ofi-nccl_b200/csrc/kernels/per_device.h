// What a process does once for each of its devices.
#pragma once
#include <atomic>
#include <stdint.h>

namespace b200 {

class OncePerDevice {
 public:
  // Runs set() unless it has succeeded for `device` before, and returns what it returns (0: success). Threads may come here at once, in
  // which case both run it; a device beyond the table has it run every time.
  template <class F>
  int run(int device, F&& set) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int rc = set();
    if (rc == 0) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace b200
