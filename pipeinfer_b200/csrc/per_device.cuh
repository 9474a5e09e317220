// per_device.cuh -- a kernel's attributes (dynamic shared memory above 48 KB, the carve-out) hold for one device: what a launch has set, per device.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>

// at the launch: static pib_per_device attrs; PIB_CHECK(attrs.once([&] { return cudaFuncSetAttribute(...); })) -- the call is made on the first launch on each device, and again for
// a larger size; an error is returned and not remembered.  Threads may make it twice, which changes nothing
class pib_per_device {
    static constexpr int DEVICES = 64;
    std::atomic<size_t> have[DEVICES];           // static objects: zero

public:
    template <typename Set> cudaError_t once(size_t size, Set set) {
        int dev = 0;
        const cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev < 0 || dev >= DEVICES) return set();
        if (have[dev].load(std::memory_order_acquire) >= size) return cudaSuccess;
        const cudaError_t r = set();
        if (r == cudaSuccess)
            for (size_t had = have[dev].load(); had < size && !have[dev].compare_exchange_weak(had, size, std::memory_order_release);) {}
        return r;
    }
    template <typename Set> cudaError_t once(Set set) { return once(1, set); }
};
