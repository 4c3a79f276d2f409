// turb_sum.cuh -- sums over a block of 256 threads.
//
// The order is that of five xor shuffles per warp (distances 16, 8, 4, 2, 1)
// and the same over the eight warps' sums.  Done with shuffles every lane
// adds at every distance: 45 FP64 warp instructions per value, which at
// GB300's two FP64 lanes per SM and clock cost more than the data of a small
// block (a dot product's 256 elements are 8).  Here the pairs of all eight
// warps are gathered in shared memory and added once each, 4 + 2 + 1 + 1 + 1
// + 3 warp instructions, the same pairs at every distance, so the sums are
// the same bits.  With this and the sums ending in the launches that form them
// (below), a step of the conjugate gradients' vector kernels went from 68 to
// 30 us at 32x16x16 and from 252 to 227 us at 256x128x128.
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

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of the blocks' partials by the block that finishes last: it adds them
// as one block of 1024 threads would (thread t takes partials t, t + 1024, ..,
// then a shuffle tree per warp and one over the warps), whatever its own
// size, so the sums do not depend on which block it is.  Partials
// [nblk, nper) are those of blocks that would have no elements: zeros, which
// adding leaves out.  nval values, value v's partials at part + v * stride.
// A launch for the sums cost 6 us at every size; this costs one round trip.
__device__ __forceinline__ bool last_block(unsigned *count, unsigned nblk)
{
    __shared__ bool last;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        last = atomicAdd(count, 1u) == nblk - 1;
        if (last) {
            *count = 0u;   // ready for the next launch
            __threadfence();
        }
    }
    __syncthreads();
    return last;
}

template <int NVAL>
__device__ __forceinline__ void sum_parts(const double *part, long long stride, int nblk, double *dst)
{
    __shared__ double sm[NVAL][1024];
    const int lt = threadIdx.y * blockDim.x + threadIdx.x, lane = lt & 31;
    if (nblk <= 256) {
        // one partial per thread of the first eight of the 32 warps: their
        // shuffle trees and one over the warps, a barrier instead of seven
#pragma unroll
        for (int v = 0; v < NVAL; v++) {
            const double r = warp_sum(lt < nblk ? __ldcg(part + v * stride + lt) : 0.0);
            if (lane == 0) sm[v][lt >> 5] = r;
        }
        __syncthreads();
        if (lt < 32) {
#pragma unroll
            for (int v = 0; v < NVAL; v++) {
                const double r = warp_sum(lane < 8 ? sm[v][lane] : 0.0);
                if (lt == 0) dst[v] = r;
            }
        }
        return;
    }
    // the 1024 threads' sums, four per thread of this block of 256
#pragma unroll
    for (int v = 0; v < NVAL; v++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            double acc = 0.0;
            // eight loads in flight, added in order: one after the other they
            // cost an L2 round trip each, 60 us for the 37000 partials of a
            // stencil kernel at 512x256x256
            for (int t = q * 256 + lt; t < nblk; t += 8 * 1024) {
                double p[8];
#pragma unroll
                for (int e = 0; e < 8; e++) p[e] = t + e * 1024 < nblk ? __ldcg(part + v * stride + t + e * 1024) : 0.0;
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (t + e * 1024 < nblk) acc += p[e];
            }
            sm[v][q * 256 + lt] = acc;
        }
    __syncthreads();
    // the trees of the 32 warps, each pair added once: warp w's entries stay
    // at w * 32 .. while their number halves (distances 16, 8, 4, 2, 1)
    if (lt < 128) {
        for (int d = 16; d >= 1; d >>= 1) {
            for (int v = 0; v < NVAL; v++)
                for (int t = lt; t < 32 * d; t += 128) {
                    const int at = (t / d) * 32 + (t & (d - 1));
                    sm[v][at] += sm[v][at + d];
                }
            asm volatile("bar.sync 2, 128;" ::: "memory");
        }
    }
    if (lt < 32) {
#pragma unroll
        for (int v = 0; v < NVAL; v++) {
            const double r = warp_sum(sm[v][lane * 32]);
            if (lt == 0) dst[v] = r;
        }
    }
}
