// gpv_once.h -- work done once per device of a process (no CUDA headers: also built by the tests).
#pragma once
#include <atomic>
#include <cstdint>

namespace gpv {

// A kernel's attributes (its dynamic shared memory above 48 KB) are set per device, so each kernel
// keeps one of these and runs its setter once for every device that launches it.  The setter is
// idempotent: threads that come at once may each run it, and none returns before it has run.  A
// setter that fails (returns false) runs again at the next launch, as one for an ordinal past 63 does.
class OncePerDevice {
 public:
  template <typename F>
  void operator()(int device, F &&set) {
    const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
    if (done_.load(std::memory_order_acquire) & bit) return;
    if (set()) done_.fetch_or(bit, std::memory_order_release);
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace gpv
