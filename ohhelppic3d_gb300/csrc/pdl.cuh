// pdl.cuh -- programmatic dependent launch: kernels of a chain that come in while the
// one before them drains.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace ohpic {
namespace {

// Waits for the kernels before this one in the stream (and their writes).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets the next kernel's CTAs come in while this one finishes.  Called late: CTAs
// let in early pile up on the SMs that happen to have room and unbalance the
// chip (a pooled solve of 64^3: 28.2 us with the call at the kernels' start, 20.6 us
// before their last stores, 32.0 us without it).
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch of clusters of `cluster` CTAs; OVERLAP: it may begin while the kernel before
// it in the stream drains (the kernel waits with pdl_wait).
template <bool OVERLAP, typename... P, typename... A>
cudaError_t launch_clusters(cudaStream_t st, dim3 grid, dim3 block, size_t smem, int cluster, void (*k)(P...),
                            A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (OVERLAP) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = (unsigned)n;
    return cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

template <typename... P, typename... A>
cudaError_t launch_overlapped(cudaStream_t st, dim3 grid, dim3 block, size_t smem, int cluster, void (*k)(P...),
                              A &&...args)
{
    return launch_clusters<true>(st, grid, block, smem, cluster, k, std::forward<A>(args)...);
}

}  // namespace
}  // namespace ohpic
