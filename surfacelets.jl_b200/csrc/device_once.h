// Per-device set-up of a kernel (function attributes, occupancy): a process may
// hold plans on several devices and call them from several threads.
#pragma once

#include <atomic>
#include <cstdint>

namespace sfl {

// Runs a set-up once a device.  Threads that come first together may each run
// it (it has to allow that); none goes on before it has been run.
class DeviceOnce {
    std::atomic<uint64_t> done_{0};

public:
    template <class F>
    void run(int device, F&& f) {
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;   // others: every time
        if (done_.load(std::memory_order_acquire) & bit) return;
        f();
        done_.fetch_or(bit, std::memory_order_release);
    }
};

}  // namespace sfl
