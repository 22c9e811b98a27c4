// What a process has been given device by device: a limit that belongs to a kernel on one device (its dynamic shared memory) is raised once for each
// device that launches the kernel, and again where a launch needs more.  Plain C++: the callers bring the device and the call that raises.
#pragma once

#include <atomic>
#include <mutex>

#define BC_KNOWN_DEVICES 64   // of any device beyond these nothing is remembered: every launch asks anew

class BcDeviceLimits {
    std::atomic<int> given[BC_KNOWN_DEVICES] = {};
    std::mutex asking;

  public:
    // raise(value), unless the device has been given as much before; its status, 0 where there was nothing to do.  One thread at a time, so that a
    // smaller value never follows a larger one.
    template <class Raise> int at_least(int device, int value, Raise&& raise) {
        if (device < 0 || device >= BC_KNOWN_DEVICES) return raise(value);
        if (given[device].load(std::memory_order_acquire) >= value) return 0;
        std::lock_guard<std::mutex> lock(asking);
        if (given[device].load(std::memory_order_relaxed) >= value) return 0;
        const int status = raise(value);
        if (status == 0) given[device].store(value, std::memory_order_release);
        return status;
    }
};
