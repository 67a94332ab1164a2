// device_once.h -- an action once per device: kernel attributes (the shared memory a
// kernel may take, its cluster size) belong to the device that is current when they are
// set, so once per process leaves every other device without them.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace msk {

class DeviceOnce {
public:
    // Runs `action` on the first call for this device; other callers return after it
    // has run.  A device beyond 63 (or unknown, negative) runs it every time.
    template <typename F>
    void run(int device, F action)
    {
        if (device < 0 || device >= 64) return action();
        const uint64_t bit = (uint64_t)1 << device;
        if (done_.load(std::memory_order_acquire) & bit) return;
        std::lock_guard<std::mutex> lk(m_);
        if (done_.load(std::memory_order_relaxed) & bit) return;
        action();
        done_.fetch_or(bit, std::memory_order_release);
    }

private:
    std::atomic<uint64_t> done_{0};
    std::mutex m_;
};

}  // namespace msk
