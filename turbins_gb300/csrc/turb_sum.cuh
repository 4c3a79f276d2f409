// turb_sum.cuh -- sums over a block of 256 threads.
//
// The order is that of five xor shuffles per warp (distances 16, 8, 4, 2, 1)
// and the same over the eight warps' sums.  Done with shuffles every lane
// adds at every distance: 45 FP64 warp instructions per value, which at
// GB300's two FP64 lanes per SM and clock cost more than the data of a small
// block (a dot product's 256 elements are 8).  Here the pairs of all eight
// warps are gathered in shared memory and added once each, 4 + 2 + 1 + 1 + 1
// + 3 warp instructions, the same pairs at every distance, so the sums are
// the same bits.  Measured at 256x128x128: see the kernels that use it.
#pragma once

// sums of NV values; the results are valid in thread 0.  Every thread of the
// block calls it; it ends without a barrier (the buffers are its own)
template <int NV>
__device__ __forceinline__ void block_sum256(const double (&v)[NV], double (&out)[NV])
{
    __shared__ double b0[NV][256], b1[NV][128];
    const int lt = threadIdx.y * blockDim.x + threadIdx.x;
    __syncthreads();   // a call before this one may still read
#pragma unroll
    for (int n = 0; n < NV; n++) b0[n][lt] = v[n];
    __syncthreads();
    if (lt < 128) {   // distance 16: (w, i) = (lt / 16, lt % 16)
        const int at = (lt >> 4) * 32 + (lt & 15);
#pragma unroll
        for (int n = 0; n < NV; n++) b1[n][lt] = b0[n][at] + b0[n][at + 16];
    }
    __syncthreads();
    if (lt < 32) {
#pragma unroll
        for (int n = 0; n < NV; n++) {
            // distance 8: 64 pairs, two per lane; distance 4: 32 pairs
            const int a0 = (lt >> 3) * 16 + (lt & 7), a1 = a0 + 64;
            const double s0 = b1[n][a0] + b1[n][a0 + 8], s1 = b1[n][a1] + b1[n][a1 + 8];
            b0[n][lt] = s0;
            b0[n][lt + 32] = s1;
            __syncwarp();
            const int at = (lt >> 2) * 8 + (lt & 3);
            double s = b0[n][at] + b0[n][at + 4];
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            // lane 4 w holds warp w's sum: the eight warps, w ^ 4, w ^ 2, w ^ 1
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            out[n] = s;
        }
    }
}
