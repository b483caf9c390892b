// Set-up that a launcher does once per device: a kernel's attributes (its opt-in to
// more than 48 KB of dynamic shared memory) hold for the device that is current when
// they are set, and a process may drive several.
#pragma once
#include <atomic>

#include <cuda_runtime.h>

namespace rh3t {

class OncePerDevice {
    static constexpr int MAX = 64; // a device beyond these is set up at every call
    std::atomic<bool> done[MAX] = {};

  public:
    // setup() until it has once returned true on device dev
    template <class F> void operator()(int dev, F setup) {
        const bool kept = dev >= 0 && dev < MAX;
        if (kept && done[dev].load(std::memory_order_acquire)) return;
        if (setup() && kept) done[dev].store(true, std::memory_order_release);
    }
};

// multiprocessors of device dev, asked for once
inline int multiprocessors(int dev) {
    constexpr int MAX = 64;
    static std::atomic<int> known[MAX] = {};
    const bool kept = dev >= 0 && dev < MAX;
    int n = kept ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 1;
    if (kept) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

} // namespace rh3t
