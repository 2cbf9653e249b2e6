// smem_limit.h -- a kernel's limit of dynamic shared memory, raised once per device.
//
// The limit belongs to the kernel on one device: remembered per process, it stayed unset for
// contexts on a second one, whose launches above 48 KB then failed.  Threads may come here
// together: raising it twice does no harm, and it counts as raised only afterwards.
#pragma once
#include <atomic>

#include <cuda_runtime_api.h>

struct SmemLimit {
    std::atomic<unsigned long long> done{ 0 };    // a bit per device (above 63: raised at every launch)

    cudaError_t raise(const void *kern, int bytes)
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
        if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
        return e;
    }
};
