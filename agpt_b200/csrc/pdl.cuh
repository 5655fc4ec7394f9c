// Programmatic dependent launch: the blocks of a kernel are placed, and what they do before pdl_wait() runs, while the kernel before it in
// the stream still works.  A step of training on few rows is a chain of some 80 short kernels; between two of them this takes the launch, the
// block start and the barrier and tensor-memory setup off the chain.
//
// Rules.  Every thread of every block calls pdl_wait() before it reads or writes device memory, before any early return: the kernel in front
// has then completed and its results are visible, and, as that kernel waited itself, so have all before it.  That goes for what was written
// long ago as well: a kernel is placed when the one in front has passed its own wait, but only a grid's own wait makes the writes of earlier
// grids visible to it.  pdl_next() comes behind pdl_wait(), so that no more than two kernels of a stream are on the device at a time and a waiting block never holds what an unplaced block of an
// earlier kernel needs.  A kernel launched in the ordinary way passes both at once, and one launched through pdl_launch behind an ordinary
// kernel, a copy or an event wait starts when that has completed.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether pdl_launch places early on this thread: on, but for the length of a call that knows better (PdlScope on its stack).  The training step and
// attention have rules by size, the optimizer launches in the ordinary way.  What is called by itself is placed early at any size: that gains up to 1.7 us, but for the
// rotation, which gains 0.3 or loses 0.6 (chains of one call, early / ordinary, us, 256, 4k, 32k, 1M rows: loss of 65 symbols 5.8 / 6.0, 6.0 / 6.3, 7.3 / 7.6, 106.8 / 107.5; embedding gradient of 128 columns
// 23.6 / 24.2, 24.8 / 25.7, 28.9 / 30.6, 173.8 / 174.5; bfloat16 store 1.1 / 1.5, 1.3 / 1.7, 4.9 / 5.1, 136.9 / 137.5; rotation of a pair 4.2 / 3.6, 3.8 / 4.1, 8.3 / 7.9, 329.3 / 329.8).
inline thread_local bool pdl_early = true;
struct PdlScope {
    const bool before;
    explicit PdlScope(bool early) : before(pdl_early) { pdl_early = early; }
    ~PdlScope() { pdl_early = before; }
    PdlScope(const PdlScope &) = delete;
};

// cluster: blocks of a cluster along x (1: none)
template <typename... P, typename... A>
static inline cudaError_t pdl_launch_clusters(void (*kernel)(P...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl_early ? 1 : 0;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = st; c.attrs = at; c.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
static inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    return pdl_launch_clusters(kernel, 1, grid, block, smem, st, static_cast<A &&>(args)...);
}
