// Launches that overlap with the end of the kernel before them in the stream (programmatic dependent launch).
//
// Between two kernels a stream leaves the GPU idle for some microseconds: the last blocks of the first end one by one, the
// second is launched, and its blocks set up barriers and tensor memory before their first load.  A kernel started by
// launch_after begins while the one before it still runs: its blocks take the places that become free, do what depends
// on no other kernel, and wait in grid_wait() until that kernel is complete and its writes are visible.
//
// With and without the attribute, device time of a pass forward and backward on one B200: linear 32 x 1024 x 1024 26.8 and
// 32.9 us, FFN 900 x 1536 x 4096 146 and 154, LayerNorm 387 x 4096 (which has nothing to set up: its launch overlaps)
// 20.6 and 25.6.  The host takes no longer for a launch either way, so a pass that is bound by the host gains nothing.
//
// Rules for a kernel that is launched this way:
//  - every thread passes grid_wait() before its first access to global memory and before it ends.  (A kernel that ended
//    without it could be complete before its predecessor, and the next one in the stream would wait for too little.)
//  - what it reads is memory that changes while the kernel is resident, behind the wait too: it is not declared
//    const __restrict__ (the compiler may move such loads across the wait) and not read by __ldg or ld.global.nc (the
//    read-only path is not kept coherent during a kernel's life, whatever waits).
//  - a kernel that takes tensor memory calls grid_trigger() behind the barrier that follows the allocation.  (Blocks of the
//    next kernel take theirs before they wait: one that came to an SM first would wait there for this kernel's end, and
//    this kernel's block for its columns, without a limit.  With all of this kernel's blocks served, none can.)
// grid_trigger() allows the next kernel's blocks to start as soon as all blocks of this one have called it or ended; it has
// no effect on what that kernel may read.  Behind any other kernel, copy or event the launch is an ordinary one.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace rb {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `cluster`: blocks of a cluster (0: none).  A failed launch is reported by the result alone: the runtime's last error is
// taken back, or the next check of another launch would report it again.
template <typename... P, typename... A>
[[nodiscard]] inline cudaError_t launch_after_clusters(void (*kern)(P...), unsigned cluster, dim3 grid, dim3 block, size_t smem,
                                                       cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = cluster ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}
template <typename... P, typename... A>
[[nodiscard]] inline cudaError_t launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                              A&&... args) {
    return launch_after_clusters(kern, 0, grid, block, smem, stream, std::forward<A>(args)...);
}

}  // namespace rb
