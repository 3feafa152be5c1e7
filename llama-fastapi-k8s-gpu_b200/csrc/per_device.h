// What has to be done once on every device, not once per process: engines on several GPUs share one process (plain C++, also built by
// host_selftest.cpp).
#pragma once
#include <atomic>
#include <stdint.h>

namespace b2 {

// One per thing to do. `set` runs on the first call for a device, and again if it failed there; calls may come from any thread (two that are first
// at once both run it).
class PerDevice {
    std::atomic<uint64_t> done{0};               // a bit per device

public:
    template <typename Set>
    bool ready(int device, Set&& set) {
        const uint64_t bit = device >= 0 && device < 64 ? (uint64_t)1 << device : 0;
        if (done.load(std::memory_order_acquire) & bit) return true;
        if (!set()) return false;
        done.fetch_or(bit, std::memory_order_release);
        return true;
    }
};

}  // namespace b2
