// How much dynamic shared memory a kernel may be launched with, beyond the 48 KB that need no asking.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime_api.h>

namespace simnets {

// The limit belongs to each device's copy of a kernel: it is raised on the current device by the first launch there, on whichever
// thread that is (backward passes launch from autograd's threads).  One object per kernel, with one `bytes`.
class SmemLimit {
public:
    template <class Kernel>
    cudaError_t raise(Kernel* kernel, int bytes) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = dev >= 0 && dev < 64 ? uint64_t(1) << dev : 0;          // (devices past the 64th: asked for at every launch)
        if (raised_.load(std::memory_order_acquire) & bit) return cudaSuccess;
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e == cudaSuccess) raised_.fetch_or(bit, std::memory_order_release);
        return e;
    }

private:
    std::atomic<uint64_t> raised_{0};
};

}  // namespace simnets
