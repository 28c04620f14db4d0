// dem_device.cuh -- what a host thread asks a device once: the blocks of a kernel it holds, after the kernel's
// shared memory has been raised there.  Kept per host thread (solvers run concurrently from threads) and per
// device: an attribute set on one device says nothing of another that the thread makes current later.
#pragma once

namespace b200dem {

constexpr int kMaxDevices = 64;   // devices past these are asked each time

struct PerDevice {
    int kept[kMaxDevices] = {};
    template <class ASK>
    int get(int dev, ASK ask) {
        if (dev < 0 || dev >= kMaxDevices) return ask(dev);
        if (kept[dev] == 0) kept[dev] = ask(dev);
        return kept[dev];
    }
};

}  // namespace b200dem
