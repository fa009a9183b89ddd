// device_once.h -- something to be done once on each device of the process (plain C++).
#pragma once
#include <atomic>
#include <stdint.h>

// A kernel's attributes belong to a device.  run(dev, set) calls set() until it has returned 0 once for this
// device; two threads that meet here may both call it, so it has to be harmless to repeat.
class DeviceOnce {
    std::atomic<uint64_t> done{0}; // a bit per device ordinal; beyond 63 every call sets

  public:
    template <typename F> int run(int dev, F set)
    {
        const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
        if (done.load(std::memory_order_acquire) & bit)
            return 0;
        const int rc = set();
        if (rc == 0)
            done.fetch_or(bit, std::memory_order_release);
        return rc;
    }
};
