// A kernel's dynamic shared memory limit, raised on every device that launches it.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace cigpu {

// cudaFuncSetAttribute acts on the current device only, so a limit raised once per
// process leaves the kernel's large launches failing on every other device. One static
// SmemLimit per kernel and launch site remembers the devices done; a failure is not
// remembered. The value is the same at every call of a site, so concurrent callers never
// lower it.
class SmemLimit {
public:
    // carveout: the preferred share of shared memory, as cudaFuncSetAttribute takes it
    template <typename K>
    cudaError_t raise(K kern, size_t bytes, int carveout = cudaSharedmemCarveoutDefault) {
        int dev = 0;
        const cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;  // past 64 devices: set at every call
        if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
        const void *k = reinterpret_cast<const void *>(kern);
        cudaError_t f = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (f == cudaSuccess && carveout != cudaSharedmemCarveoutDefault)
            f = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
        if (f == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
        return f;
    }

private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace cigpu
