// turb_conv.cuh -- BF16 tensor-core 3x3x3 convolutions (k_conv.cu) used by
// the pressure-guess network (k_net.cu).
//
// Activation layout ("channel-blocked"): a tensor of C channels on an
// X x Y x Z voxel grid is stored as [C/8][Z][Y][X][8] BF16, i.e. C/8 planes
// of 16-byte vectors: 16-byte copies build the K-major operand rows of the
// forward and data-gradient convolutions, and a TMA box lands in shared memory
// as [kc/8][voxel][8], the MN-major operand (voxels = K) of the weight gradient.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "turb_internal.cuh"

typedef __nv_bfloat16 bf16;

// which kernel runs one convolution on one grid, and its weight layout
struct ConvPlan {
    int rows;    // 1: row-ring kernel (cin, cout <= 32), else the tap-staged one
    int zring;   // row-ring kernel: the ring runs along z (X < 128), else along y
    int kc;      // tap-staged kernel: channels per K chunk
};
ConvPlan conv_plan(int X, int Y, int Z, int cin, int cout);

// Epilogue options of a convolution: out = mask?( relu?( acc + bias ) )
// and, for at most 16 channels in and out, an optional 1x1x1 head hout = headw . out + headb
struct ConvEpi {
    const float *bias = nullptr;
    int relu = 0;
    const bf16 *mask = nullptr;
    bf16 *out = nullptr;
    const float *headw = nullptr;
    const float *headb = nullptr;
    float *hout = nullptr;
};

// Weight packs: W[27][cout][cin] FP32 -> the B operand of the forward
// convolution and of the data-gradient convolution (taps mirrored, cin and
// cout exchanged), in the layout of the kernel each plan selects.
void conv_pack_weights(cudaStream_t s, const float *W, int cin, int cout, const ConvPlan &pf, const ConvPlan &pb,
                       bf16 *wf, bf16 *wd);

// elements of a weight pack buffer for a conv of (cin, cout) on any grid (both
// layouts pad K to 128-byte rows); buffers start zeroed
inline long long conv_pack_elems(int cin, int cout)
{
    long long wide = 27LL * ((cin + 31) / 32) * cout * 64;
    long long rows = 3LL * ((3 * cin + 63) / 64) * 3 * cout * 64;
    return wide > rows ? wide : rows;
}

int conv3_fwd(cudaStream_t s, const bf16 *in, int X, int Y, int Z, int cin, int cout, const bf16 *wpk,
              const ConvEpi &e, int *err, int nsm, int pdl);
int conv3_wgrad(cudaStream_t s, const bf16 *x, const bf16 *dy, int X, int Y, int Z, int cin, int cout, float *dw,
                int *err, int nsm, int pdl);
int conv_selftest_umma(int mn_major, int swap, unsigned long long *mismatches);
const char *conv_last_error();

// A network kernel starts while the one before it on the stream drains (pdl):
// its set-up (barriers, TMEM, resident weights) overlaps that kernel's tail.
// Every such kernel calls pdl_trigger and, before it reads or writes anything
// the others do, pdl_wait; the first kernel of a pass is an ordinary launch,
// so what was written before the pass is visible to all
template <typename K, typename... A>
inline void net_launch(int pdl, K k, int gx, int gy, int threads, uint32_t smem, cudaStream_t s, A... args)
{
    launch_early(pdl, k, dim3((unsigned)gx, (unsigned)gy), dim3((unsigned)threads), smem, s, args...);
}
