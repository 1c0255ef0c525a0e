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

// A launch that may begin while the kernel before it in the stream drains.
template <typename... P, typename... A>
cudaError_t launch_overlapped(cudaStream_t st, dim3 grid, dim3 block, size_t smem, int cluster, void (*k)(P...),
                              A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

}  // namespace
}  // namespace ohpic
