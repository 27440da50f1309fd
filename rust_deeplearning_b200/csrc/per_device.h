// What a launcher has to raise once for every device: the opt-in to more shared memory holds for the device that is current.
#pragma once

#include <atomic>
#include <mutex>

class RdlRaisedPerDevice {
    static constexpr int DEVICES = 64;
    std::atomic<int> most_[DEVICES] = {};            // what each device has been raised to
    std::mutex raising_;

public:
    // f() -> 0 where it succeeded; run when `value` is above what the device has been raised to, by one thread at a time, and again
    // where it failed (each time for a device there is no place for).
    template <typename F>
    int run(int device, int value, F f) {
        if (device < 0 || device >= DEVICES) return f();
        if (most_[device].load(std::memory_order_acquire) >= value) return 0;
        std::lock_guard<std::mutex> hold(raising_);
        if (most_[device].load(std::memory_order_relaxed) >= value) return 0;
        const int e = f();
        if (e == 0) most_[device].store(value, std::memory_order_release);
        return e;
    }
};
