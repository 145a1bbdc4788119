// What has to be set up once per device of a process (the opt-in to more than 48 KB of dynamic shared memory belongs to a function ON a
// device): one bit per device ordinal.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime_api.h>

namespace sg {

// Calls `set` (which returns whether it succeeded) unless it has succeeded for `dev` before; ordinals past the bits are set every time.
template <typename F> bool once_per_device(std::atomic<uint64_t>& done, int dev, F&& set) {
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (!set()) return false;
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

inline int current_device() {
    int dev = 0;
    cudaGetDevice(&dev);
    return dev;
}

// SMs of the current device; the answers are kept per ordinal, a launcher asks several times per launch
inline int device_sms() {
    static std::atomic<int> known[64];
    const int dev = current_device(), k = dev >= 0 && dev < 64 ? dev : -1;
    int n = k >= 0 ? known[k].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) return 148;
        if (k >= 0) known[k].store(n, std::memory_order_relaxed);
    }
    return n;
}

}  // namespace sg
