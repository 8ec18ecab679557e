// Settings that belong to a device, made once for each: a kernel's attributes (its dynamic shared memory beyond
// 48 KB above all) are those of the module loaded on the current device.
#pragma once

#include <atomic>

#include "common.cuh"

namespace cdftb {

// run(f) calls f, which returns a cdftb status, unless it has succeeded on the current device before. Threads that
// come first together may each call it: f sets the same values every time. Costs a cudaGetDevice (tens of ns).
class OncePerDevice {
    std::atomic<unsigned long long> done_{0};  // a bit per device; devices from 64 on are set every time

public:
    template <typename F>
    int run(F&& f) {
        int device = 0;
        int st = check(cudaGetDevice(&device));
        if (st != CDFTB_OK) return st;
        const unsigned long long bit = device < 64 ? 1ull << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return CDFTB_OK;
        st = f();
        if (st == CDFTB_OK) done_.fetch_or(bit, std::memory_order_release);
        return st;
    }
};

}  // namespace cdftb
