// dynamic_smem.h -- the dynamic shared memory that kernels are allowed.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <mutex>

namespace tgl {

// A kernel's largest dynamic shared memory is an attribute of the function in
// the current device's context, shared by every world and thread that uses
// it: raise it when a launch needs more, and never lower it below what another
// world (or an earlier plan, whose captured graphs may still launch) needs.
// It is read back each time: a second device, or a device that was reset, has
// the 48 KB default.
inline void allow_dynamic_smem(const void *kernel, size_t bytes) {
    static std::mutex lock;
    if (bytes <= 40 * 1024) return;  // with any static share within the default
    std::lock_guard<std::mutex> guard(lock);
    cudaFuncAttributes now{};
    if (cudaFuncGetAttributes(&now, kernel) == cudaSuccess && (size_t)now.maxDynamicSharedSizeBytes < bytes)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// The same for a kernel that is launched too often to ask each time (0.8 us of
// the host's): what each device was granted is kept, which does not outlive a
// reset of the device.
struct DynamicSmem {
    static constexpr int DEVICES = 64;
    std::atomic<size_t> granted[DEVICES] = {};

    void allow(const void *kernel, size_t bytes) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) return;
        if (device < DEVICES && granted[device].load() >= bytes) return;
        allow_dynamic_smem(kernel, bytes);
        size_t seen = device < DEVICES ? granted[device].load() : bytes;
        while (seen < bytes && !granted[device].compare_exchange_weak(seen, bytes)) {
        }
    }
};

}  // namespace tgl
