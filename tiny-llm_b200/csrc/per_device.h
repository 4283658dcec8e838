// Something set up once on every device it is used on: a kernel's attributes belong to the device that is current when they are set.
#pragma once

#include <atomic>
#include <cstdint>

namespace tl {

class PerDevice {
  public:
    // true: `set` has succeeded on `device`, now or before.  A failure is not remembered, the next call tries again.
    template <typename Set>
    bool operator()(int device, Set set) {
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;  // of further devices: set on every call
        if (done_.load(std::memory_order_acquire) & bit) return true;
        if (!set()) return false;
        done_.fetch_or(bit, std::memory_order_release);
        return true;
    }

  private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace tl
