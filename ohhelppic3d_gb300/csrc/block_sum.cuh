// block_sum.cuh -- FP64 sums of a whole grid of 256-thread blocks.
#pragma once
#include <cuda_runtime.h>

namespace ohpic {

// Adds the block's sum of each of v[0..N) to out[0..N), one atomic per block: with
// one per warp, the atomics on the same few words took most of a reduction of a
// million particles (a diagnostics call at 32^3 x 16 ppc, FP32: 270 -> 113 us).
template <int N>
__device__ __forceinline__ void block_sum_add(double (&v)[N], double *const (&out)[N])
{
    __shared__ double part[N][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) part[k][warp] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += part[threadIdx.x][w];
        double *p = out[0];
#pragma unroll
        for (int k = 1; k < N; ++k)
            if ((int)threadIdx.x == k) p = out[k];
        atomicAdd(p, s);
    }
}

}  // namespace ohpic
