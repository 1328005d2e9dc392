// once_per_device.h -- set-up calls that hold for the process and a device.
#pragma once
#include <atomic>
#include <cstdint>

namespace falcon {

// Calls set() until it has returned 0 (success) for a device once; a failure is returned
// and tried again by the next call. Devices from 64 on are set every time. Threads that
// come at once may each call set().
class OncePerDevice {
    std::atomic<uint64_t> done_{0};

  public:
    template <class F> auto operator()(int device, F set) {
        using E = decltype(set());
        const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return E{};
        const E e = set();
        if (e == E{}) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace falcon
