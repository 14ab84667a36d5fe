// Kernel launches that overlap their own launch latency with the kernel in front of them on the stream (programmatic dependent
// launch).  Small layers are chains of kernels of 2 to 10 us; without this the GPU idles a microsecond or more between two of
// them, and as long again while the next grid's blocks start up.
//
// Rule: a kernel launched this way calls stream_order() before it touches memory.  That waits until the kernels in front have
// finished and their writes are visible; nothing about stream order changes.
//
// The next grid's blocks come up as this one's leave, not earlier.  Asking for them on entry (griddepcontrol.launch_dependents) put
// blocks that only wait beside the running ones and changed on which multiprocessors the blocks of the next kernel land.  With /
// without it, us: 1357 images through the 3x32x32 network 1235 / 1211, its training step at 2048 4782 / 4724 and at 256 763 / 767,
// at 12 in float64 730 / 712; 256 instances over 4x2x2 blocks of 256 x 256 x 32 x 32: 4786 / 4689, of which the forward pass
// 1005 / 920 (923 with plain launches).
#pragma once
#include <cuda_runtime.h>
#include <utility>
#include "smem_limit.hpp"

namespace simnets {

__device__ __forceinline__ void stream_order() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class Kernel>
struct DependentLaunch {
    Kernel* kernel;
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
    int cluster;                                        // CTAs per cluster along the grid's y (which it divides)
    template <class... Args>
    void operator()(Args&&... args) const {
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = attr[1].val.clusterDim.z = 1;
        attr[1].val.clusterDim.y = unsigned(cluster);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = cluster > 1 ? 2 : 1;
        cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);         // (a failure is what cudaGetLastError returns next)
    }
};

template <class Kernel>
DependentLaunch<Kernel> in_stream_order(Kernel* kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster = 1) {
    return {kernel, grid, block, smem, stream, cluster};
}

}  // namespace simnets
