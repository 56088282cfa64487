// Set-up that a device needs once before a kernel can be launched on it (function attributes belong to a device, so a
// process that drives several GPUs repeats it for each).  Plain C++, so that the host test can compile it alone.
#pragma once

#include <atomic>
#include <mutex>

// run(device, setup): setup() returns 0 or an error code.  No call returns 0 before one setup() of that device has
// succeeded (threads that arrive meanwhile wait for it), and one that failed is tried again by the next call.
class B200PerDeviceOnce {
public:
    template <typename F>
    int run(int device, F setup) {
        if (device < 0 || device >= 64) return setup();
        const unsigned long long bit = 1ull << device;
        if (done_.load(std::memory_order_acquire) & bit) return 0;
        std::lock_guard<std::mutex> lock(mutex_);
        if (done_.load(std::memory_order_relaxed) & bit) return 0;
        const int st = setup();
        if (st == 0) done_.fetch_or(bit, std::memory_order_release);
        return st;
    }

private:
    std::atomic<unsigned long long> done_{0};
    std::mutex mutex_;
};
