// Work that has to be done once on every device of the process, by whichever call comes first there: raising a kernel's
// shared-memory limit, say, which holds for the device that is current.
#pragma once

#include <atomic>
#include <cstdint>

namespace psx {

class OncePerDevice {
public:
    // Returns what work() returns, 0 (success) where it has succeeded before.  Work that fails is tried again by the next
    // call; two threads that come at the same time may both do it, and devices from 64 on do it every time.
    template <class Work>
    auto run(int device, Work work) -> decltype(work()) {
        const bool noted = device >= 0 && device < 64;
        const uint64_t bit = noted ? uint64_t(1) << device : 0;
        if ((done_.load(std::memory_order_acquire) & bit) != 0) return decltype(work())(0);
        const auto result = work();
        if (result == decltype(work())(0)) done_.fetch_or(bit, std::memory_order_release);
        return result;
    }

private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace psx
