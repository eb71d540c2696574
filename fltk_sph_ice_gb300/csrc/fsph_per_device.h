/*
 * fsph_per_device.h -- what has to be done once on each device of a process.
 *
 * A kernel's dynamic shared-memory limit belongs to the device that was current
 * when it was raised: a process that goes on to another device has to raise it
 * there again.  No CUDA in here, so that it can be tested without a device.
 */
#pragma once
#include <mutex>

namespace fsph {

class PerDevice {
public:
    static constexpr int kDevices = 64; /* past it: done at every call */

    /* what `act` gave on device `dev`: it is called at the first call for a device and
     * again after it failed (gave false).  Safe from several threads. */
    template <class Act>
    bool once(int dev, Act &&act) {
        if (dev < 0 || dev >= kDevices) return act();
        std::lock_guard<std::mutex> lock(mu_);
        if (!done_[dev]) done_[dev] = act();
        return done_[dev];
    }

private:
    std::mutex mu_;
    bool done_[kDevices] = {};
};

}  // namespace fsph
