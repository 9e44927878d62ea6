// nb_scan.cuh -- prefix sums within a warp and a block.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace nb {

__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive block scan of one value per thread; returns the block total in *total.
__device__ __forceinline__ int block_excl_scan(int v, int* sh_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int inc = warp_incl_scan(v);
    if (lane == 31) sh_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nw ? sh_warp[lane] : 0;
        const int wi = warp_incl_scan(w);
        if (lane < nw) sh_warp[lane] = wi - w;
        if (lane == nw - 1) sh_warp[32] = wi;
    }
    __syncthreads();
    const int r = sh_warp[warp] + inc - v;
    *total = sh_warp[32];
    __syncthreads();
    return r;
}

}  // namespace nb
