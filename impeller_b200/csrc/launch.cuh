// Kernel launches that follow one another closely.
//
// A chain of kernels of a few microseconds each pays for every hand-over: the
// next kernel is only set up once the previous one has drained.  launch_next
// lets it be set up as soon as the previous kernel's blocks have ended
// (programmatic stream serialization); grid_wait, the first thing such a kernel
// does, waits until the previous kernel has completed and its writes are
// visible.  That orders ordinary accesses as a plain launch does.  It does not
// order loads through the read-only path (__ldg, or const __restrict__
// parameters): the compiler may take those ahead of the wait, and the hardware
// wants their data unwritten from the kernel's start, which now lies before the
// previous kernel's end.  So such a kernel reads with plain loads whatever a
// kernel of the chain writes; only inputs that none of them writes
// (descriptors, the point array) may be const __restrict__.
//
// No kernel asks for its successor earlier (griddepcontrol.launch_dependents).
// Blocks that are set up while others still run hold registers and shared
// memory that other streams' kernels could use, and crowd onto the SMs that
// have room.  With that request at the start of every kernel, three streams of
// 10^5-point BLS12-381 MSMs took 1183 us an MSM (953 without), a transform of
// 2^18 elements 87 us (65) and a lone MSM of 300 points 216 us (210).
#pragma once

#include <cuda_runtime.h>

namespace impeller {

__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// kern<<<grid, block, smem, st>>>(args...) for a kernel that starts with grid_wait.
template <class... P, class... A>
inline cudaError_t launch_next(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// The same with the blocks in clusters of `cluster`.
template <class... P, class... A>
inline cudaError_t launch_cluster(void (*kern)(P...), dim3 grid, dim3 block, unsigned cluster, cudaStream_t st,
                                  A... args) {
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace impeller
