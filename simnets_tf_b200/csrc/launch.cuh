// Kernel launches that overlap their own launch latency with the kernel in front of them on the stream (programmatic dependent
// launch).  Small layers are chains of kernels of 2 to 10 us; without this the GPU idles a microsecond or more between two of
// them, and as long again while the next grid's blocks start up.
//
// Rules: a kernel launched this way calls stream_order() before it touches memory.  That waits until the kernels in front have
// finished and their writes are visible, and only then lets the next one start up, so that at most one grid waits behind the
// running one; nothing else about stream order changes.
#pragma once
#include <cuda_runtime.h>
#include <utility>
#include "smem_limit.hpp"

namespace simnets {

__device__ __forceinline__ void stream_order() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class Kernel>
struct DependentLaunch {
    Kernel* kernel;
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
    template <class... Args>
    void operator()(Args&&... args) const {
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);         // (a failure is what cudaGetLastError returns next)
    }
};

template <class Kernel>
DependentLaunch<Kernel> in_stream_order(Kernel* kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream) { return {kernel, grid, block, smem, stream}; }

}  // namespace simnets
