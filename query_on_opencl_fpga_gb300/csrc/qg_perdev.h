// qg_perdev.h -- what a call site has set up on each device of the process.
#pragma once
#include <stdint.h>

#include <atomic>

// A kernel's attributes belong to a device, so "set already" is kept per device: the
// largest value set there, 0 for none.  For objects with static storage; threads may
// race, and then set the same thing twice.  Devices beyond the table are set each time.
struct qg_per_device {
    static constexpr int DEVICES = 64;
    std::atomic<uint64_t> have[DEVICES];

    bool covers(int device, uint64_t value) const {
        return device >= 0 && device < DEVICES && have[device].load(std::memory_order_acquire) >= value;
    }
    void set(int device, uint64_t value) {
        if (device < 0 || device >= DEVICES) return;
        uint64_t old = have[device].load(std::memory_order_relaxed);
        while (old < value && !have[device].compare_exchange_weak(old, value, std::memory_order_release)) {
        }
    }
};
