// Work that a process does once per device, such as a kernel's opt-in to more shared memory (a function attribute belongs to the device that was
// current when it was set).  Any number of threads and devices; plain C++.
#pragma once
#include <atomic>

namespace jsm {

struct DeviceOnce {
    std::atomic<unsigned long long> done{0};  // a bit per device
    // step() on the first call for `device` that succeeds (returns 0), and on every call for a device beyond 63; two threads may both run it
    template <typename Step>
    int run(int device, Step step) {
        const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;
        if (done.load(std::memory_order_acquire) & bit) return 0;
        const int status = step();
        if (status == 0) done.fetch_or(bit, std::memory_order_release);
        return status;
    }
};

}  // namespace jsm
