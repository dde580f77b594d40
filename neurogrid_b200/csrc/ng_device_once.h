// Something that belongs to a device and is to be done once for each (a kernel's shared-memory limit: a process may use one
// device after another).  Plain C++.
#pragma once
#include <atomic>

// `done`: one bit a device, zero at first.  Runs `f` if it has not succeeded for `device` before; false if it fails now.  Two
// threads may both run it, which is harmless for what is set to the same value.
template <typename F>
static inline bool ng_once_per_device(std::atomic<unsigned long long>& done, int device, F f) {
    const unsigned long long bit = 1ull << (device & 63);
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (!f()) return false;
    done.fetch_or(bit, std::memory_order_release);
    return true;
}
