// Sums over the threads of a CTA.
#pragma once
#include <stdint.h>

namespace nq {

// exclusive sum over the CTA's threads (whole warps, at most 1,024 threads) and the total; every thread takes part.
// s_warp: 32 ints
__device__ __forceinline__ int cta_exclusive_sum(int v, int* s_warp, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();                      // s_warp may still be read from an earlier sum
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
    }
    total = __shfl_sync(0xffffffffu, w, 31);
    const int before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);      // sum of the earlier warps
    return inc - v + (warp ? before : 0);
}

}  // namespace nq
