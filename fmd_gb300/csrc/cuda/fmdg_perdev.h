// An answer that belongs to a device (what it has room for, an attribute set
// on it), asked for once per device and kept for the process.  Two threads
// that ask at the same time both get it from `ask`, which gives the same
// each time.
#pragma once

#include <atomic>

class PerDevice
{
    static constexpr int MAX_DEVICES = 64;
    std::atomic<int> kept[MAX_DEVICES] = {};       // 0: not asked yet

public:
    // ask(): a positive number, with `device` meant by its caller
    template <typename F>
    int get(int device, F &&ask)
    {
        if (device < 0 || device >= MAX_DEVICES) return ask();
        int v = kept[device].load(std::memory_order_acquire);
        if (v == 0)
        {
            v = ask();
            kept[device].store(v, std::memory_order_release);
        }
        return v;
    }
};
