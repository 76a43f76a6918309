// The limit of dynamic shared memory a kernel may be launched with, per device: it stays with the function, so a launch that needs
// no more than was granted before skips the call.  Several threads may launch one kernel with different sizes: the limit
// is looked at again, set and noted under a lock, so that it only ever grows.
#pragma once

#include <atomic>
#include <mutex>

struct TqSmemGrant {
    static constexpr int kDevices = 64;
    std::mutex lock;
    std::atomic<int> granted[kDevices] = {};

    // `set` raises the limit to its argument and returns 0, or an error, which is handed on.
    template <class Set>
    int raise(int device, int bytes, Set set) {
        std::atomic<int>& limit = granted[device & (kDevices - 1)];
        if (limit.load(std::memory_order_acquire) >= bytes) return 0;
        std::lock_guard<std::mutex> hold(lock);
        if (limit.load(std::memory_order_relaxed) >= bytes) return 0;
        const int error = set(bytes);
        if (error == 0) limit.store(bytes, std::memory_order_release);
        return error;
    }
};
