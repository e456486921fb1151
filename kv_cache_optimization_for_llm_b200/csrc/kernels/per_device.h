// Something that has to be done once on every device, such as a kernel's limit of shared memory, which a launcher of a process with engines
// on several devices must not remember for all of them.  Plain C++.
#pragma once

#include <atomic>

class OncePerDevice {
 public:
  // f() (0: done) unless it has been done on this device; devices beyond the 64th, and none (-1), are not remembered.
  template <class F>
  auto operator()(int device, F f) -> decltype(f()) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
    using R = decltype(f());
    if (done_.load(std::memory_order_acquire) & bit) return R(0);
    const R rc = f();
    if (rc == R(0)) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<unsigned long long> done_{0};
};
