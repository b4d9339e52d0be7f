// Host-side helpers that the launchers share.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace mf {

// Dynamic shared memory above 48 KiB has to be allowed once per kernel and device, always with the same size for a kernel.
// Safe for threads that launch for the first time together, and for a process that uses several GPUs.
template <auto KERNEL>
inline bool AllowSmem(size_t bytes)
{
    static std::atomic<bool> allowed[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        (void)cudaGetLastError();
        return false;
    }
    if (!allowed[dev].load(std::memory_order_relaxed)) {
        if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        allowed[dev].store(true, std::memory_order_relaxed);
    }
    return true;
}

}  // namespace mf
