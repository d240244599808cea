// A step that is taken once on each device: a kernel's attributes and the
// sizes of the device itself hold for the device that is current when they are
// set or read, and one process may use several.  A step that throws is taken
// again by the next caller.
#pragma once

#include <stdint.h>

#include <atomic>
#include <mutex>
#include <stdexcept>

namespace gb {

static constexpr int kMaxDevices = 64;

class device_once {
    std::atomic<uint64_t> done{0};
    std::mutex mu;

public:
    template <class F>
    void run(int device, F step)
    {
        if (device < 0 || device >= kMaxDevices) throw std::out_of_range("device index out of range");
        const uint64_t bit = (uint64_t)1 << device;
        if (done.load(std::memory_order_acquire) & bit) return;
        std::lock_guard<std::mutex> lk(mu);
        if (done.load(std::memory_order_relaxed) & bit) return;
        step();
        done.fetch_or(bit, std::memory_order_release);
    }
};

}  // namespace gb
