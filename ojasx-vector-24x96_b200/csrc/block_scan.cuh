// Exclusive prefix sum of one int per thread over a block of up to 1024 threads.
#pragma once

namespace ojx {

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_tot /* [33] shared */, int* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    int inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
    }
    __syncthreads();   // warp_tot may still be read from the previous scan
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int t = lane < nwarp ? warp_tot[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, t, off);
            if (lane >= off) t += o;
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    *total = warp_tot[nwarp - 1];
    return inc - v + (wid > 0 ? warp_tot[wid - 1] : 0);
}

}  // namespace ojx
