// What a process keeps per device about its launches.  A kernel's limit of dynamic shared memory as it has been raised so far: the limit
// belongs to a device's copy of the kernel, so a process that launches on a second GPU has to raise it there too.  Plain C++ (the calls that
// ask for the current device and set the limit are the caller's), any number of threads.
#pragma once

#include <atomic>
#include <mutex>
#include <stddef.h>

namespace pb {

class DeviceLimit {
public:
    // Makes sure that the current device's limit is at least `bytes`.  device(int*) gives the current device, raise(size_t)
    // sets its limit; both return 0 or an error, which is returned.  A limit is never lowered: a smaller request than one
    // before does nothing, so a launch that follows never finds less than it asked for.
    template <typename Device, typename Raise>
    int allow(size_t bytes, Device device, Raise raise) {
        int dev = 0;
        if (const int rc = device(&dev)) return rc;
        if (dev < 0 || dev >= kDevices) return raise(bytes);        // more devices than are kept account of
        if (held_[dev].load(std::memory_order_acquire) >= bytes) return 0;
        std::lock_guard<std::mutex> guard(lock_);
        if (held_[dev].load(std::memory_order_relaxed) >= bytes) return 0;
        if (const int rc = raise(bytes)) return rc;
        held_[dev].store(bytes, std::memory_order_release);
        return 0;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<size_t> held_[kDevices] = {};
    std::mutex lock_;
};

// A number above 0 that belongs to a device and is asked for once on each: how many of a launch's clusters it holds, say.
class DeviceCount {
public:
    // The number of `dev`, the current device, or 0 where it cannot be had; that is not remembered, so the next call asks again.
    // ask(int*) gives the number and returns 0 or an error.
    template <typename Ask>
    int get(int dev, Ask ask) {
        int n = 0;
        const bool kept = dev >= 0 && dev < kDevices;               // more devices than are kept account of are asked every time
        if (kept) n = known_[dev].load(std::memory_order_relaxed);
        if (n > 0) return n;
        if (ask(&n) != 0 || n <= 0) return 0;
        if (kept) known_[dev].store(n, std::memory_order_relaxed);
        return n;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<int> known_[kDevices] = {};
};

}  // namespace pb
