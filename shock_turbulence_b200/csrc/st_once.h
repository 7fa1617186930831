// st_once.h - an action that a kernel needs once on each device.
#pragma once
#include <atomic>
#include <cstdint>

namespace st {

// Runs set() (0: done, otherwise an error) on the first call for each device
// and on every call until one has succeeded; returns what it returned.  Callers
// on several threads may run it at the same time, so that it has to leave the
// same state whoever comes last.  Devices beyond kDevices run it on every call.
class OncePerDevice {
    static constexpr int kDevices = 64;
    std::atomic<uint64_t> done_{0};

  public:
    template <class Set>
    int operator()(int dev, Set set) {
        const uint64_t bit = dev >= 0 && dev < kDevices ? (uint64_t)1 << dev : 0;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        const int e = set();
        if (e == 0) done_.fetch_or(bit, std::memory_order_release);
        return e;
    }
};

}  // namespace st
