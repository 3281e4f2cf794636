// The opt-in of one kernel to dynamic shared memory beyond 48 KB, per device: it only ever grows. Contexts on one device share it and
// may be used from several threads, so that a smaller request must neither overtake nor undo a larger one.
#pragma once
#include <atomic>
#include <mutex>
#include <stddef.h>

struct SmemOptIn {
    std::mutex m;
    std::atomic<size_t> have[64] = {};
    // set(bytes) makes the opt-in and returns 0 when it worked; whatever else it returns is passed on and not remembered
    template <class F>
    int raise(int device, size_t want, F set) {
        std::atomic<size_t>& h = have[device & 63];
        if (h.load(std::memory_order_acquire) >= want) return 0;
        std::lock_guard<std::mutex> lock(m);
        if (h.load(std::memory_order_relaxed) >= want) return 0;
        const int e = set(want);
        if (e == 0) h.store(want, std::memory_order_release);
        return e;
    }
};
