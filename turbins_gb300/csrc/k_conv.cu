// k_conv.cu -- 3x3x3 convolutions (stride 1, zero padding 1) as implicit
// GEMMs on the tcgen05 tensor cores: BF16 operands, FP32 accumulators in
// TMEM, four producer warps, one MMA thread and four epilogue warps per CTA,
// persistent CTAs.
//
// Forward (and data gradient, the same kernel on mirrored weights):
//   out[v][co] = sum_tap sum_ci W[tap][co][ci] * in[v + off(tap)][ci]
// GEMM view: M = 128 voxels, N = output channels, K = taps x cin.  Two kernels:
// k_conv_rows (cin, cout <= 32: resident weights, taps of one axis stacked
// along N) and k_conv_wide (more channels: weights staged per tap, the output
// channels split over CTAs where there are few tiles).  Both read 128-byte
// swizzled K-major operands and load a voxel row once for its three x taps.
// Against one load per tap into unswizzled operands (a K step then took 150-230
// cycles whatever N is, and a 16-byte-wide box one cycle per voxel) and a row
// kernel that formed its descriptors at run time, the network's forward pass
// went from 329 to 190 us at 64x32x32 and from 1318 to 704 us at 256x128x128.
//
// Weight gradient: dW[tap][co][ci] = sum_v dy[v][co] * in[v + off(tap)][ci];
// M = (taps of a group) x cin = 128 rows, N = cout, K = voxels, both operands
// MN-major straight from the channel-blocked layout.  Each CTA accumulates a
// range of voxel tiles in TMEM and adds its partial sums to FP32 dW.
#include <cstdio>
#include <cstring>
#include <mutex>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "tc_ptx.cuh"
#include "turb_conv.cuh"
#include "turb_internal.cuh"

namespace {

char g_conv_err[256] = "";

// barrier waits that must outlive an abort: copies and MMAs in flight
__device__ __forceinline__ void settle(uint32_t bar, uint32_t parity)
{
    volatile int never = 0;
    tc::mbar_wait(bar, parity, &never);
}

__device__ __forceinline__ void fail(volatile int *abort_, int *err, int code)
{
    *abort_ = 1;
    atomicExch(err, code);
}

// last fill of stage s among `n` fills of an S-stage ring, waited for so that
// no copy is still landing when the CTA exits
__device__ __forceinline__ void drain(uint32_t bars, int base, uint32_t n, int S)
{
    for (int s = 0; s < S; s++) {
        if ((uint32_t)s >= n) break;
        uint32_t last = (uint32_t)s + (uint32_t)S * ((n - 1 - (uint32_t)s) / (uint32_t)S);
        settle(bars + 8 * (base + s), (last / S) & 1);
    }
}

// what is done to 16 output channels of one voxel: bias, ReLU, mask, BF16
// store, optional 1x1x1 head (hsum)
struct EpiP {
    const float *bias;
    int relu;
    const bf16 *mask;
    bf16 *out;
    const float *headw, *headb;
    float *hout;
    size_t plane;
};

__device__ __forceinline__ void epilogue16(const EpiP &a, int ch, const uint32_t (&rr)[16], const float (&bias)[16],
                                           const float (&hw)[16], size_t vox, float &hsum)
{
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(rr[j]) + bias[j];
    const size_t o0 = ((size_t)(2 * ch) * a.plane + vox) * 8, o1 = o0 + a.plane * 8;
    if (a.relu) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = fmaxf(v[j], 0.f);
    }
    if (a.mask) {
        uint4 m0 = *reinterpret_cast<const uint4 *>(a.mask + o0);
        uint4 m1 = *reinterpret_cast<const uint4 *>(a.mask + o1);
        const bf16 *p0 = reinterpret_cast<const bf16 *>(&m0), *p1 = reinterpret_cast<const bf16 *>(&m1);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (!(__bfloat162float(p0[j]) > 0.f)) v[j] = 0.f;
            if (!(__bfloat162float(p1[j]) > 0.f)) v[8 + j] = 0.f;
        }
    }
    uint4 w0, w1;
    bf16 *q0 = reinterpret_cast<bf16 *>(&w0), *q1 = reinterpret_cast<bf16 *>(&w1);
#pragma unroll
    for (int j = 0; j < 8; j++) { q0[j] = __float2bfloat16_rn(v[j]); q1[j] = __float2bfloat16_rn(v[8 + j]); }
    if (a.out) {
        *reinterpret_cast<uint4 *>(a.out + o0) = w0;
        *reinterpret_cast<uint4 *>(a.out + o1) = w1;
    }
    if (a.headw) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            hsum = fmaf(hw[j], __bfloat162float(q0[j]), hsum);
            hsum = fmaf(hw[8 + j], __bfloat162float(q1[j]), hsum);
        }
    }
}

// 128-byte-swizzle K-major operand at saddr (8-row groups 1024 bytes apart);
// the swizzle follows the absolute address, so shifted starts need no offset
__host__ __device__ inline uint64_t sw128_desc(uint32_t saddr)
{
    return tc::sdesc(saddr, 16, 1024) | (2ull << 61);
}

// 128-byte-swizzle MN-major operand: rows of 64 M (or N) elements, one K each;
// the next 64 elements `atom` bytes on
__host__ __device__ inline uint64_t mn128_desc(uint32_t saddr, uint32_t atom)
{
    return tc::sdesc(saddr, atom, 1024) | (2ull << 61);
}

__device__ __forceinline__ void tmem_st16_zero(uint32_t taddr)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
        "%1};" ::"r"(taddr),
        "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int SROWS = 136;                 // voxel rows of 128 bytes in a slot, SUSED of them read
constexpr int SUSED = 130;
constexpr uint32_t SBYTES = SROWS * 128;   // a multiple of 1024

// ---- row-ring convolution (cin, cout <= 32) ----------------------------------------
// Axes: x; the ring axis r (y where X >= 128, else z); the stack axis q (the
// other one).  A CTA takes items of 128 consecutive positions of the (q, x)
// line times a run of consecutive r.  The line holds a padding position either
// side of each q's X voxels unless X is a multiple of 128, so that short x
// extents fill the 128 rows of an MMA too.
// Operands use the 128-byte-swizzle K-major layout, the one the tensor core
// fetches fastest: every shared-memory row is one voxel holding 64 K elements,
// here the channels of its three q planes (K = dq * cin + ci, zero padded),
// 16-byte chunk c of row p stored at chunk c ^ (p % 8).  One r of the line (130
// voxel rows, from position s0 - 1) is a ring slot, filled by 16-byte cp.async
// (producer warp L % 4 loads slot L).  The A operand of tap dx is the slot
// shifted by dx rows; dq and the channels are the K steps.  Input r feeds the
// outputs r+1, r, r-1 (dr = 0, 1, 2): the weights of the three dr taps are
// stacked along N, so one MMA (M = 128 voxels, N = 3 cout, K = 16) per dx and
// K step covers all of them; the three targets are consecutive blocks of a
// TMEM ring of NBLK accumulator blocks (block of output v = NBLK-1 - v mod
// NBLK, so r+1, r, r-1 are ascending; a wrap splits the MMA).  Accumulation is
// always on: the epilogue zeroes a block as soon as it has read it.  Weights
// are resident.  Order of the sums: dr, dx, dq where X >= 128; dr, dq, dx
// below.
constexpr int RING = 4;   // ring slots
constexpr int NBLK = 8;   // TMEM accumulator blocks

struct RowArgs {
    int X, W;             // voxels and positions per q of the line
    int R, rs, Q, qs;     // ring and stack axis: extent, voxels between neighbours
    int ntx, rch, nitems; // line tiles, r per item
    const bf16 *in, *wpk;
    EpiP epi;
    int *err;
};

constexpr int rows_nkb(int cin) { return (3 * cin + 63) / 64; }
// resident weights of the row kernel: per dx and K block, 3 cout rows of 128 bytes
constexpr uint32_t rows_wbytes(int cin, int cout) { return 3u * (uint32_t)rows_nkb(cin) * 3u * (uint32_t)cout * 128u; }
constexpr uint32_t rows_smem(int cin, int cout)
{
    return RING * (uint32_t)rows_nkb(cin) * SBYTES + rows_wbytes(cin, cout) + 1024u;
}

// barrier slots of k_conv_rows
constexpr int RF = 0, RE = RING, BRDY = 2 * RING, BFREE = 2 * RING + NBLK, RWB = 2 * RING + 2 * NBLK,
              RFIN = RWB + 1, RNBAR = RWB + 2;

__device__ __forceinline__ uint32_t blk_of(uint32_t v) { return NBLK - 1 - v % NBLK; }

template <int CIN, int COUT, int ZRING>
__global__ void __launch_bounds__(288) k_conv_rows(const RowArgs a)
{
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t bar[RNBAR];
    __shared__ uint32_t tslot;
    __shared__ int abort_s;
    constexpr int NKB = rows_nkb(CIN);
    constexpr int NKG = CIN / 8;           // channel blocks of 8
    constexpr int NREAL = 3 * NKG;         // real 16-byte chunks per voxel row (3 q planes)
    constexpr uint32_t SLOT = NKB * SBYTES;
    constexpr uint32_t NCOLS = NBLK * COUT;
    volatile int *abort_ = &abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t sS = (tc::smem_u32(dsm) + 1023u) & ~1023u;   // slot ring
    const uint32_t sW = sS + RING * SLOT;                       // resident stacked weights
    const uint32_t bars = tc::smem_u32(bar);

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int i = 0; i < RNBAR; i++) {
            uint32_t cnt = 1;
            if (i >= RF && i < RF + RING) cnt = 32;             // the producer warp of the slot
            if (i >= BFREE && i < BFREE + NBLK) cnt = 4;        // epilogue warps
            tc::mbar_init(bars + 8 * i, cnt);
        }
        tc::mbar_fence_init();
    }
    if (warp == 8) {
        tc::tmem_alloc(tc::smem_u32(&tslot), NCOLS);
        tc::tmem_relinquish();
    }
    if (warp >= 4 && warp < 8) {   // K padding chunks of the slots are never loaded: zero them once
        uint8_t *g = dsm + (sS - tc::smem_u32(dsm));
        constexpr int NPAD = 8 * NKB - NREAL;
        for (int i = threadIdx.x - 128; i < RING * SROWS * NPAD; i += 128) {
            const int c = NREAL + i % NPAD, r = i / NPAD, p = r % SROWS, slot = r / SROWS;
            *reinterpret_cast<uint4 *>(g + (uint32_t)slot * SLOT + (uint32_t)(c >> 3) * SBYTES + (uint32_t)p * 128u +
                                       (uint32_t)(((c & 7) ^ (p & 7)) << 4)) = make_uint4(0, 0, 0, 0);
        }
        tc::fence_proxy_async();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    pdl_trigger();   // with the TMEM taken: the next kernel's blocks wait for what is left of it
    const uint32_t tbase = tslot;
    if (warp < 4) {   // accumulators start at zero
        for (uint32_t c = 0; c < NCOLS; c += 16) tmem_st16_zero(tbase + ((uint32_t)(warp * 32) << 16) + c);
        tmem_wait_st();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();

    if (warp >= 4 && warp < 8) {
        // ---- producers
        const int pw = warp - 4;
        if (pw == 0 && lane == 0) {
            tc::mbar_expect_tx(bars + 8 * RWB, rows_wbytes(CIN, COUT));
            tc::bulk_load(sW, a.wpk, rows_wbytes(CIN, COUT), bars + 8 * RWB);
        }
        pdl_wait();   // the weights were packed before the kernel ahead of this one began
        const uint32_t sbase = sS + (uint32_t)pw * SLOT;
        uint32_t L = 0;
        bool ok = true;
        for (int it = blockIdx.x; ok && it < a.nitems; it += gridDim.x) {
            const int s0 = (it % a.ntx) * 128, rb = (it / a.ntx) * a.rch, nr = min(a.rch, a.R - rb);
            // this lane's voxel rows: position, plane, which of the planes q-1, q, q+1 exist
            const bf16 *src[5];
            uint32_t have[5];
#pragma unroll
            for (int i = 0; i < 5; i++) {
                const int p = lane + 32 * i;
                int q, x;
                if (a.W == a.X) {
                    q = s0 / a.X;
                    x = s0 - q * a.X - 1 + p;
                } else {
                    const int s = s0 - 1 + p;
                    q = s < 0 ? 0 : s / a.W;
                    x = s < 0 ? -1 : s - q * a.W - 1;
                }
                const bool v = p < SUSED && x >= 0 && x < a.X && q < a.Q;
                src[i] = a.in + (v ? ((size_t)q * a.qs + x) * 8 : 0);
                have[i] = v ? (q > 0 ? 1u : 0u) | 2u | (q + 1 < a.Q ? 4u : 0u) : 0u;
            }
            for (int j = 0; j < nr + 2; j++, L++) {
                if ((int)(L & 3u) != pw) continue;
                if (L >= RING && !tc::mbar_wait(bars + 8 * (RE + pw), ((L / RING) & 1u) ^ 1u, abort_)) {
                    ok = false;
                    break;
                }
                // chunk c = dq * NKG + cb of voxel row p comes from channel block cb
                // of plane q + dq - 1; zero outside the grid
                const int rr = rb - 1 + j;
                const bool rok = rr >= 0 && rr < a.R;
                const long long ro = (long long)(rok ? rr : 0) * a.rs;
#pragma unroll
                for (int c = 0; c < NREAL; c++) {
                    constexpr int G = NKG;
                    const int d = c / G, cb = c % G;
                    const long long co = ((long long)cb * (long long)a.epi.plane + ro + (long long)(d - 1) * a.qs) * 8;
                    const uint32_t rdst = sbase + (uint32_t)(c >> 3) * SBYTES + (uint32_t)lane * 128u +
                                          (uint32_t)(((c & 7) ^ (lane & 7)) << 4);
#pragma unroll
                    for (int i = 0; i < 5; i++) {
                        if (i == 4 && lane >= SUSED - 128) continue;
                        const bool v = rok && (have[i] >> d & 1u);
                        cp_async16(rdst + 4096u * i, v ? src[i] + co : a.in, v ? 16u : 0u);
                    }
                }
                cp_async_commit();
                cp_async_wait<0>();
                tc::fence_proxy_async();
                tc::mbar_arrive(bars + 8 * (RF + pw));
            }
        }
        cp_async_wait<0>();
        if (!ok) fail(abort_, a.err, 3);
        if (pw == 0 && lane == 0) settle(bars + 8 * RWB, 0);
    } else if (warp == 8) {
        if (lane == 0) {
            constexpr uint32_t WREG = 3u * COUT * 128u;   // weights of one (dx, K block)
            constexpr uint32_t IDESC0 = tc::idesc_bf16(128, 0, 0, 0);
            const uint64_t wdesc = sw128_desc(sW), sdesc0 = sw128_desc(sS);
            uint32_t L = 0, V = 0;
            bool ok = tc::mbar_wait(bars + 8 * RWB, 0, abort_);
            // taps k0 .. k0+n-1 of the input slot into n consecutive blocks from b0
            auto issue = [&](uint32_t slot, uint32_t k0, uint32_t n, uint32_t b0) {
                const uint32_t idesc = IDESC0 + ((n * COUT >> 3) << 17), dt = tbase + b0 * COUT;
                const uint64_t ad0 = sdesc0 + slot * (SLOT >> 4), bd0 = wdesc + k0 * (COUT * 128u >> 4);
#pragma unroll
                for (int e = 0; e < 9 * (CIN / 16); e++) {
                    constexpr int NC = CIN / 16;
                    const int dx = ZRING ? e / NC % 3 : e / (3 * NC), ks = ZRING ? e / (3 * NC) * NC + e % NC : e % (3 * NC);
                    const uint32_t ao = (uint32_t)(ks >> 2) * SBYTES + (uint32_t)dx * 128u + (uint32_t)(ks & 3) * 32u;
                    const uint32_t bo = (uint32_t)(dx * NKB + (ks >> 2)) * WREG + (uint32_t)(ks & 3) * 32u;
                    tc::mma_bf16(dt, ad0 + (ao >> 4), bd0 + (bo >> 4), idesc, 1u);
                }
            };
            for (int it = blockIdx.x; ok && it < a.nitems; it += gridDim.x) {
                const int rb = (it / a.ntx) * a.rch, nr = min(a.rch, a.R - rb);
                for (int j = 0; j < nr + 2; j++, L++) {
                    if (j < nr) {   // output j is touched for the first time
                        const uint32_t g = V + (uint32_t)j;
                        if (!tc::mbar_wait(bars + 8 * (BFREE + blk_of(g)), ((g / NBLK) & 1u) ^ 1u, abort_)) { ok = false; break; }
                    }
                    const uint32_t slot = L % RING;
                    if (!tc::mbar_wait(bars + 8 * (RF + slot), (L / RING) & 1u, abort_)) { ok = false; break; }
                    tc::fence_after();
                    // outputs j, j-1, j-2 (k = dr) that exist: taps k0 .. k1-1, their blocks
                    // ascending from output j - k0 up to a wrap
                    const uint32_t k0 = j < nr ? 0u : (uint32_t)(j - nr + 1), k1 = j < 2 ? (uint32_t)j + 1u : 3u;
                    const uint32_t b0 = blk_of(V + (uint32_t)j - k0);
                    const uint32_t n1 = min(k1 - k0, (uint32_t)NBLK - b0);
                    issue(slot, k0, n1, b0);
                    if (n1 < k1 - k0) issue(slot, k0 + n1, k1 - k0 - n1, 0u);
                    tc::mma_commit(bars + 8 * (RE + slot));                                            // input slot done
                    if (j >= 2) tc::mma_commit(bars + 8 * (BRDY + blk_of(V + (uint32_t)(j - 2))));     // output j-2 done
                }
                V += (uint32_t)nr;
            }
            if (!ok) fail(abort_, a.err, 3);
            tc::mma_commit(bars + 8 * RFIN);
            settle(bars + 8 * RFIN, 0);
        }
    } else if (warp < 4) {
        // ---- epilogue: read each output's block, zero it, store the voxels
        const int row = warp * 32 + lane;
        pdl_wait();
        float bias[COUT / 16][16], hw[16];
#pragma unroll
        for (int c = 0; c < COUT; c++) bias[c / 16][c % 16] = a.epi.bias ? a.epi.bias[c] : 0.f;
#pragma unroll
        for (int c = 0; c < 16; c++) hw[c] = a.epi.headw ? a.epi.headw[c] : 0.f;
        const float hb = a.epi.hout ? *a.epi.headb : 0.f;
        uint32_t V = 0;
        bool ok = true;
        for (int it = blockIdx.x; ok && it < a.nitems; it += gridDim.x) {
            const int s = (it % a.ntx) * 128 + row, rb = (it / a.ntx) * a.rch, nr = min(a.rch, a.R - rb);
            const int q = s / a.W, x = s - q * a.W - (a.W == a.X ? 0 : 1);
            const bool valid = q < a.Q && x >= 0 && x < a.X;
            size_t vox = (size_t)q * a.qs + x + (size_t)rb * a.rs;
            for (int j = 0; j < nr; j++, vox += a.rs) {
                const uint32_t g = V + (uint32_t)j, b = blk_of(g);
                if (!__all_sync(0xffffffffu, tc::mbar_wait(bars + 8 * (BRDY + b), (g / NBLK) & 1u, abort_))) { fail(abort_, a.err, 3); ok = false; break; }
                tc::fence_after();
                const uint32_t taddr = tbase + ((uint32_t)(warp * 32) << 16) + b * COUT;
                uint32_t rr[COUT / 16][16];
#pragma unroll
                for (int ch = 0; ch < COUT / 16; ch++) tc::tmem_ld16(taddr + (uint32_t)ch * 16u, rr[ch]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int ch = 0; ch < COUT / 16; ch++) tmem_st16_zero(taddr + (uint32_t)ch * 16u);
                tmem_wait_st();
                tc::fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(bars + 8 * (BFREE + b));
                if (!valid) continue;
                float hsum = 0.f;
#pragma unroll
                for (int ch = 0; ch < COUT / 16; ch++) epilogue16(a.epi, ch, rr[ch], bias[ch], hw, vox, hsum);
                if (a.epi.hout) a.epi.hout[vox] = hsum + hb;
            }
            V += (uint32_t)nr;
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 8) tc::tmem_dealloc(tbase, NCOLS);
}

// ---- tap-staged convolution (more channels) ------------------------------------------
// A tile is 128 consecutive positions of the line (z, y, x) with a padding
// position either side of each x row, and nt of the output channels.  A stage
// is one (channel chunk, dz, dy): the 130 voxel rows of the line at that offset
// (up to 64 channels, 128-byte-swizzled K-major rows, zero outside the grid)
// and the weights of its three dx taps.  The A operand of tap dx is the stage
// shifted by dx rows, so a voxel row is loaded 9 times instead of 27.  Four
// producer warps keep two stages in flight behind the one they fill; the
// accumulator is double buffered.  Order of the sums: chunk, dz, dy, dx, channel.
struct WideArgs {
    int X, Y, Z, W;
    int cin, cout, kc, nkc, nt, nsplit;
    int ntiles, stages;
    uint32_t stride;
    const bf16 *in, *wpk;
    EpiP epi;
    int *err;
};
constexpr int WSTAGES = 8, WLAG = 2;
// barrier slots: A full, weights full, stage empty, accumulator full / empty
constexpr int WFA = 0, WFB = WSTAGES, WE = 2 * WSTAGES, WAF = 3 * WSTAGES, WAE = WAF + 2, WFIN = WAE + 2, WNBAR = WFIN + 1;

// position s of the padded line: voxel (x, y, z); false on a padding position or past the end
__device__ __forceinline__ bool line_at(int s, int W, int X, int Y, int Z, int &x, int &y, int &z)
{
    if (s < 0) { x = y = z = 0; return false; }
    const int r = s / W;
    x = s - r * W - 1;
    z = r / Y;
    y = r - z * Y;
    return x >= 0 && x < X && z < Z;
}

__global__ void __launch_bounds__(288) k_conv_wide(const WideArgs a)
{
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t bar[WNBAR];
    __shared__ uint32_t tslot;
    __shared__ int abort_s;
    volatile int *abort_ = &abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s0 = (tc::smem_u32(dsm) + 1023u) & ~1023u;
    const uint32_t bars = tc::smem_u32(bar);
    uint32_t ncols = 32;
    while (ncols < 2u * (uint32_t)a.nt) ncols <<= 1;
    const int nwork = a.ntiles * a.nsplit, nst = 9 * a.nkc;

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int i = 0; i < WNBAR; i++)
            tc::mbar_init(bars + 8 * i, i < WFB ? 128u : (i == WAE || i == WAE + 1) ? 4u : 1u);
        tc::mbar_fence_init();
    }
    if (warp == 8) {
        tc::tmem_alloc(tc::smem_u32(&tslot), ncols);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    pdl_trigger();
    const uint32_t tbase = tslot;
    const uint32_t S = (uint32_t)a.stages;

    if (warp >= 4 && warp < 8) {
        // ---- producers: thread t loads voxel row t; the first 16 also a chunk of rows 128, 129
        const int t = threadIdx.x - 128;
        const int p2 = 128 + (t >> 3), c2 = t & 7;
        uint32_t u = 0, slot = 0, par = 1;          // fills issued; slot u % S and its empty parity
        uint32_t aslot = 0;                         // slot of the next fill to report
        bool ok = true;
        pdl_wait();
        for (int w = blockIdx.x; ok && w < nwork; w += gridDim.x) {
            const int tile = w / a.nsplit, n0 = (w - tile * a.nsplit) * a.nt;
            int x, y, z, x2, y2, z2;
            const bool v = line_at(tile * 128 - 1 + t, a.W, a.X, a.Y, a.Z, x, y, z);
            const bool v2 = t < 16 && line_at(tile * 128 - 1 + p2, a.W, a.X, a.Y, a.Z, x2, y2, z2);
            const long long vox = v ? ((long long)z * a.Y + y) * a.X + x : 0;
            const long long vox2 = v2 ? ((long long)z2 * a.Y + y2) * a.X + x2 : 0;
            for (int st = 0; st < nst; st++, u++) {
                if (!tc::mbar_wait(bars + 8 * (WE + slot), par, abort_)) { ok = false; break; }
                const int kci = st / 9, e = st - kci * 9, dz = e / 3 - 1, dy = e % 3 - 1;
                const uint32_t buf = s0 + slot * a.stride;
                if (t == 0) {   // three dx taps' weights of the nt channels
                    const uint32_t bytes = (uint32_t)a.nt * 128u;
                    tc::mbar_expect_tx(bars + 8 * (WFB + slot), 3u * bytes);
                    for (int dx = 0; dx < 3; dx++)
                        tc::bulk_load(buf + SBYTES + (uint32_t)dx * bytes,
                                      a.wpk + ((size_t)(st * 3 + dx) * a.cout + n0) * 64, bytes, bars + 8 * (WFB + slot));
                }
                const int nch = min(a.kc, a.cin - kci * a.kc) >> 3;   // 16-byte chunks of this channel chunk
                const long long off = ((long long)dz * a.Y + dy) * a.X, cb0 = (long long)kci * (a.kc >> 3);
                {
                    const bool in = v && z + dz >= 0 && z + dz < a.Z && y + dy >= 0 && y + dy < a.Y;
                    const bf16 *src = in ? a.in + (cb0 * (long long)a.epi.plane + vox + off) * 8 : a.in;
                    const long long step = in ? (long long)a.epi.plane * 8 : 0;
                    const uint32_t dst = buf + (uint32_t)t * 128u, sw = (uint32_t)(t & 7), n16 = in ? 16u : 0u;
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        if (c < nch) cp_async16(dst + (((uint32_t)c ^ sw) << 4), src + c * step, n16);
                }
                if (t < 16 && c2 < nch) {
                    const bool in = v2 && z2 + dz >= 0 && z2 + dz < a.Z && y2 + dy >= 0 && y2 + dy < a.Y;
                    cp_async16(buf + (uint32_t)p2 * 128u + (uint32_t)((c2 ^ (p2 & 7)) << 4),
                               in ? a.in + ((cb0 + c2) * (long long)a.epi.plane + vox2 + off) * 8 : a.in, in ? 16u : 0u);
                }
                cp_async_commit();
                if (u >= WLAG) {
                    cp_async_wait<WLAG>();
                    tc::fence_proxy_async();
                    tc::mbar_arrive(bars + 8 * (WFA + aslot));
                    if (++aslot == S) aslot = 0;
                }
                if (++slot == S) { slot = 0; par ^= 1u; }
            }
        }
        cp_async_wait<0>();
        tc::fence_proxy_async();
        for (uint32_t i = u > WLAG ? u - WLAG : 0u; i < u; i++) {
            tc::mbar_arrive(bars + 8 * (WFA + aslot));
            if (++aslot == S) aslot = 0;
        }
        if (!ok) fail(abort_, a.err, 1);
        if (t == 0) drain(bars, WFB, u, (int)S);
    } else if (warp == 8) {
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_bf16(128, a.nt, 0, 0);
            const uint32_t bstep = (uint32_t)a.nt * 128u >> 4;
            uint32_t slot = 0, par = 0, it = 0;
            bool ok = true;
            for (int w = blockIdx.x; ok && w < nwork; w += gridDim.x, it++) {
                const uint32_t ab = it & 1u;
                if (!tc::mbar_wait(bars + 8 * (WAE + ab), ((it >> 1) & 1u) ^ 1u, abort_)) { ok = false; break; }
                const uint32_t dt = tbase + ab * (uint32_t)a.nt;
                for (int st = 0; st < nst; st++) {
                    if (!tc::mbar_wait(bars + 8 * (WFB + slot), par, abort_) ||
                        !tc::mbar_wait(bars + 8 * (WFA + slot), par, abort_)) { ok = false; break; }
                    tc::fence_after();
                    const uint64_t ad = sw128_desc(s0 + slot * a.stride), bd = ad + (SBYTES >> 4);
                    const int nks = min(a.kc, a.cin - st / 9 * a.kc) >> 4;
#pragma unroll
                    for (int dx = 0; dx < 3; dx++)
#pragma unroll
                        for (int ks = 0; ks < 4; ks++)
                            if (ks < nks)
                                tc::mma_bf16(dt, ad + (uint32_t)(dx * 8 + ks * 2), bd + (uint32_t)dx * bstep + (uint32_t)(ks * 2),
                                             idesc, (st | dx | ks) != 0);
                    tc::mma_commit(bars + 8 * (WE + slot));
                    if (++slot == S) { slot = 0; par ^= 1u; }
                }
                if (ok) tc::mma_commit(bars + 8 * (WAF + ab));
            }
            if (!ok) fail(abort_, a.err, 1);
            tc::mma_commit(bars + 8 * WFIN);
            settle(bars + 8 * WFIN, 0);
        }
    } else if (warp < 4) {
        const float none[16] = {};
        uint32_t it = 0;
        pdl_wait();
        for (int w = blockIdx.x; w < nwork; w += gridDim.x, it++) {
            const int tile = w / a.nsplit, n0 = (w - tile * a.nsplit) * a.nt;
            int x, y, z;
            const bool valid = line_at(tile * 128 + warp * 32 + lane, a.W, a.X, a.Y, a.Z, x, y, z);
            const size_t vox = valid ? ((size_t)z * a.Y + y) * a.X + x : 0;
            const uint32_t ab = it & 1u;
            if (!__all_sync(0xffffffffu, tc::mbar_wait(bars + 8 * (WAF + ab), (it >> 1) & 1u, abort_))) { fail(abort_, a.err, 1); break; }
            tc::fence_after();
            const uint32_t taddr = tbase + ((uint32_t)(warp * 32) << 16) + ab * (uint32_t)a.nt;
            float hsum = 0.f;
            for (int ch = 0; ch < (a.nt >> 4); ch++) {
                uint32_t rr[16];
                tc::tmem_ld16(taddr + (uint32_t)ch * 16u, rr);
                float bias[16];
#pragma unroll
                for (int j = 0; j < 16; j++) bias[j] = a.epi.bias ? a.epi.bias[n0 + ch * 16 + j] : 0.f;
                tc::tmem_wait_ld();
                if (valid) epilogue16(a.epi, (n0 >> 4) + ch, rr, bias, none, vox, hsum);
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bars + 8 * (WAE + ab));
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 8) tc::tmem_dealloc(tbase, ncols);
}


// ---- weight gradient --------------------------------------------------------------
struct WgArgs {
    int X, Y, Z, cin, cout, G, ngroups, nsplit;
    int bx, by, bz, nb, ntx, nty, ntz, ntiles;
    uint32_t tapbytes, bbytes, stride;
    float *dw;
    int *err;
};

constexpr int WG_STAGES = 3;

__global__ void __launch_bounds__(192) k_wgrad(const __grid_constant__ CUtensorMap mapX,
                                               const __grid_constant__ CUtensorMap mapD, WgArgs a)
{
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t bar[2 * WG_STAGES + 2];
    __shared__ uint32_t tslot;
    __shared__ int abort_s;
    volatile int *abort_ = &abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s0 = (tc::smem_u32(dsm) + 1023u) & ~1023u;
    const uint32_t bars = tc::smem_u32(bar);
    const int F = 0, E = WG_STAGES, DONE = 2 * WG_STAGES, FINB = 2 * WG_STAGES + 1;
    const uint32_t ncols = a.cout < 32 ? 32u : (uint32_t)a.cout;
    const int g = blockIdx.x % a.ngroups, sp = blockIdx.x / a.ngroups;
    const int ntaps = min(a.G, 27 - g * a.G);

    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int i = 0; i < 2 * WG_STAGES + 2; i++) tc::mbar_init(bars + 8 * i, 1);
        tc::mbar_fence_init();
        tc::prefetch_map(&mapX);
        tc::prefetch_map(&mapD);
    }
    if (warp == 1) {
        tc::tmem_alloc(tc::smem_u32(&tslot), ncols);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    pdl_trigger();
    pdl_wait();
    const uint32_t tbase = tslot;
    const uint32_t sbo = (uint32_t)a.nb * 16u;   // next 8 channels
    const int nks = a.nb >> 4;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t u = 0;
            bool ok = true;
            for (int t = sp; t < a.ntiles; t += a.nsplit) {
                int tx = t % a.ntx, r = t / a.ntx, ty = r % a.nty, tz = r / a.nty;
                int x0 = tx * a.bx, y0 = ty * a.by, z0 = tz * a.bz;
                uint32_t s = u % WG_STAGES;
                if (!tc::mbar_wait(bars + 8 * (E + s), ((u / WG_STAGES) & 1u) ^ 1u, abort_)) { ok = false; break; }
                uint32_t buf = s0 + s * a.stride;
                tc::mbar_expect_tx(bars + 8 * (F + s), (uint32_t)ntaps * a.tapbytes + a.bbytes);
                for (int tl = 0; tl < ntaps; tl++) {
                    int tap = g * a.G + tl, dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
                    tc::tma_load5(buf + (uint32_t)tl * a.tapbytes, &mapX, 0, x0 + dx - 1, y0 + dy - 1, z0 + dz - 1, 0,
                                  bars + 8 * (F + s));
                }
                tc::tma_load5(buf + (uint32_t)a.G * a.tapbytes, &mapD, 0, x0, y0, z0, 0, bars + 8 * (F + s));
                u++;
            }
            if (!ok) fail(abort_, a.err, 2);
            drain(bars, F, u, WG_STAGES);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_bf16(128, a.cout, 1, 1);
            uint32_t u = 0;
            bool ok = true;
            for (int t = sp; t < a.ntiles; t += a.nsplit) {
                uint32_t s = u % WG_STAGES;
                if (!tc::mbar_wait(bars + 8 * (F + s), (u / WG_STAGES) & 1u, abort_)) { ok = false; break; }
                tc::fence_after();
                uint32_t abuf = s0 + s * a.stride, bbuf = abuf + (uint32_t)a.G * a.tapbytes;
                for (int ks = 0; ks < nks; ks++) {
                    uint64_t ad = tc::sdesc(abuf + (uint32_t)ks * 256u, 128, sbo);
                    uint64_t bd = tc::sdesc(bbuf + (uint32_t)ks * 256u, 128, sbo);
                    tc::mma_bf16(tbase, ad, bd, idesc, (u | (uint32_t)ks) != 0);
                }
                tc::mma_commit(bars + 8 * (E + s));
                u++;
            }
            if (!ok) fail(abort_, a.err, 2);
            tc::mma_commit(bars + 8 * DONE);
            tc::mma_commit(bars + 8 * FINB);
            tc::mbar_wait(bars + 8 * FINB, 0, abort_);
        }
    } else if (warp >= 2) {
        const int q = warp & 3, row = q * 32 + lane;
        const bool have = sp < a.ntiles;
        if (have) {
            if (!tc::mbar_wait(bars + 8 * DONE, 0, abort_)) {
                fail(abort_, a.err, 2);
            } else {
                tc::fence_after();
                const int tl = row / a.cin, ci = row % a.cin, tap = g * a.G + tl;
                const bool valid = tl < ntaps && !*abort_;
                uint32_t taddr = tbase + ((uint32_t)(q * 32) << 16);
                for (int ch = 0; ch < (a.cout >> 4); ch++) {
                    uint32_t rr[16];
                    tc::tmem_ld16(taddr + (uint32_t)ch * 16u, rr);
                    tc::tmem_wait_ld();
                    if (!valid) continue;
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        atomicAdd(a.dw + ((size_t)tap * a.cout + ch * 16 + j) * a.cin + ci, __uint_as_float(rr[j]));
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 1) tc::tmem_dealloc(tbase, ncols);
}

// ---- weight gradient, few channels (cin, cout <= 32) ---------------------------------
// dW[tap][co][ci] by steps of RA rows of x of a 128-position line tile (lines,
// ring axis r and stack axis q as in k_conv_rows).  Both operands are
// MN-major, 128-byte swizzled: a shared-memory row is one voxel (K), holding
// for A the channels of its three q planes of each of the RA rows (M =
// (row, dq, ci), 128 with padding), for B the gradients of the rows around
// them (N = (t, co), t = 0 .. RA + 1 from the row before the first).  Tap dx is
// a shift of A by dx rows, so a step is 3 x 8 MMAs, one accumulator per dx; row
// a and t belong to tap dr = a - t + 2.  On large grids a CTA has one dx and
// three times the steps: the FP32 accumulation chains then stay as long as
// k_wgrad's, and the gradients within 2e-5 of its sums.  A box per tap of an unswizzled layout
// (k_wgrad) loads a 16-byte voxel row per cycle and 27 of them per voxel:
// 141 us at 128x64x64, 16 -> 16 channels, against 33 us here; 37, 41 and 26 us
// against 13, 17 and 18 us for 32 -> 16, 32 -> 32 and 16 -> 32 at 64x32x32.
template <int CIN>
struct WgR {
    static constexpr int RA = CIN == 16 ? 2 : 1, NB = RA + 2;   // rows of x and of dy a step holds
};
struct WgRowArgs {
    int X, W, R, rs, Q, qs, cstep;   // cstep: voxels of the grid (between channel blocks)
    int ntx, nsteps, zring, ndx;     // ndx: x taps per CTA, 3 or 1
    const bf16 *x, *dy;
    float *dw;
    int *err;
};
constexpr int WRS = 3;   // stages
constexpr int wgr_batoms(int cin, int cout) { return ((cin == 16 ? 4 : 3) * cout + 63) / 64; }
constexpr uint32_t wgr_stage(int cin, int cout) { return 2u * SBYTES + (uint32_t)wgr_batoms(cin, cout) * 16384u; }

template <int CIN, int COUT>
__global__ void __launch_bounds__(288) k_wgrad_rows(const WgRowArgs a)
{
    constexpr int RA = WgR<CIN>::RA, NB = WgR<CIN>::NB, N = NB * COUT, GA = CIN / 8, GB = COUT / 8;
    constexpr uint32_t STAGE = wgr_stage(CIN, COUT), NCOLS = 3 * N <= 256 ? 256 : 512;
    constexpr int FA_ = 0, EM_ = WRS, DONE = 2 * WRS, NB_ = DONE + 1;
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t bar[NB_];
    __shared__ uint32_t tslot;
    __shared__ int abort_s;
    volatile int *abort_ = &abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s0 = (tc::smem_u32(dsm) + 1023u) & ~1023u;
    const uint32_t bars = tc::smem_u32(bar);
    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int i = 0; i < NB_; i++) tc::mbar_init(bars + 8 * i, i < WRS ? 128u : 1u);
        tc::mbar_fence_init();
    }
    if (warp == 8) {
        tc::tmem_alloc(tc::smem_u32(&tslot), NCOLS);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    pdl_trigger();
    pdl_wait();
    const uint32_t tbase = tslot;
    const int nrow = (a.R + RA - 1) / RA;   // steps per line tile
    const int ng = 3 / a.ndx, dx0 = blockIdx.x % ng, dx1 = dx0 + a.ndx, w0 = blockIdx.x / ng, wstep = gridDim.x / ng;

    if (warp >= 4 && warp < 8) {
        // ---- producers: thread t loads voxel row t of both operands; the first
        // also a chunk of A's rows 128, 129
        constexpr int CA = RA * 3 * GA, CB = NB * GB;   // chunks of a voxel row
        const int t = threadIdx.x - 128;
        const int p2 = 128 + t / CA, e2 = t % CA;
        uint32_t u = 0, slot = 0, par = 1, aslot = 0;
        bool ok = true;
        auto place = [&](int s, int &q, int &x) {
            if (a.W == a.X) { q = s < 0 ? -1 : s / a.X; x = s - q * a.X; }
            else { q = s < 0 ? -1 : s / a.W; x = s - q * a.W - 1; }
            return q >= 0 && q < a.Q && x >= 0 && x < a.X;
        };
        for (int w = w0; w < a.nsteps; w += wstep, u++) {
            if (!tc::mbar_wait(bars + 8 * (EM_ + slot), par, abort_)) { ok = false; break; }
            const int tile = w / nrow, r0 = (w - tile * nrow) * RA, line0 = tile * 128;
            const uint32_t buf = s0 + slot * STAGE;
            int q, x, q2, x2, qb, xb;
            bool v = place(line0 - 1 + t, q, x), v2 = t < 2 * CA && place(line0 - 1 + p2, q2, x2);
            const bool vb = place(line0 + t, qb, xb);
            if (a.W == a.X) {   // a tile lies within one q: its halo positions are outside the grid or in it
                const int qt = line0 / a.X, xt = line0 - qt * a.X;
                q = qt; x = xt - 1 + t; v = x >= 0 && x < a.X;
                q2 = qt; x2 = xt - 1 + p2; v2 = t < 2 * CA && x2 < a.X;
            }
            auto load_a = [&](int p, int e, bool pv, int pq, int px) {
                const int ra = e / (3 * GA), d = e / GA % 3, cb = e % GA, rr = r0 + ra, qq = pq + d - 1;
                const bool in = pv && rr < a.R && qq >= 0 && qq < a.Q;
                // M index of the chunk: row a at 64 a where two rows share an operand
                const int k8 = (RA == 2 ? ra * 8 : 0) + d * GA + cb;
                const uint32_t dst = buf + (uint32_t)(k8 >> 3) * SBYTES + (uint32_t)p * 128u + (uint32_t)(((k8 & 7) ^ (p & 7)) << 4);
                cp_async16(dst, in ? a.x + ((long long)cb * a.cstep + (long long)rr * a.rs + (long long)qq * a.qs + px) * 8 : a.x,
                           in ? 16u : 0u);
            };
#pragma unroll
            for (int e = 0; e < CA; e++) load_a(t, e, v, q, x);
            if (t < 2 * CA) load_a(p2, e2, v2, q2, x2);
#pragma unroll
            for (int e = 0; e < CB; e++) {
                const int tt = e / GB, cb = e % GB, rr = r0 - 1 + tt;
                const bool in = vb && rr >= 0 && rr < a.R;
                const uint32_t dst = buf + 2u * SBYTES + (uint32_t)(e >> 3) * 16384u + (uint32_t)t * 128u +
                                     (uint32_t)(((e & 7) ^ (t & 7)) << 4);
                cp_async16(dst, in ? a.dy + ((long long)cb * a.cstep + (long long)rr * a.rs + (long long)qb * a.qs + xb) * 8 : a.dy,
                           in ? 16u : 0u);
            }
            cp_async_commit();
            if (u >= 1) {
                cp_async_wait<1>();
                tc::fence_proxy_async();
                tc::mbar_arrive(bars + 8 * (FA_ + aslot));
                if (++aslot == WRS) aslot = 0;
            }
            if (++slot == WRS) { slot = 0; par ^= 1u; }
        }
        cp_async_wait<0>();
        tc::fence_proxy_async();
        if (u > 0) tc::mbar_arrive(bars + 8 * (FA_ + aslot));
        if (!ok) fail(abort_, a.err, 2);
    } else if (warp == 8) {
        if (lane == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16(128, N, 1, 1);
            uint32_t slot = 0, par = 0, u = 0;
            bool ok = true;
            for (int w = w0; w < a.nsteps; w += wstep, u++) {
                if (!tc::mbar_wait(bars + 8 * (FA_ + slot), par, abort_)) { ok = false; break; }
                tc::fence_after();
                const uint32_t buf = s0 + slot * STAGE;
                const uint64_t ad = mn128_desc(buf, SBYTES), bd = mn128_desc(buf + 2u * SBYTES, 16384u);
#pragma unroll
                for (int dx = 0; dx < 3; dx++)
                    if (dx >= dx0 && dx < dx1)
#pragma unroll
                    for (int ks = 0; ks < 8; ks++)
                        tc::mma_bf16(tbase + (uint32_t)(dx * N), ad + (uint32_t)(dx * 8 + ks * 128), bd + (uint32_t)(ks * 128),
                                     idesc, u > 0 || ks > 0);
                tc::mma_commit(bars + 8 * (EM_ + slot));
                if (++slot == WRS) { slot = 0; par ^= 1u; }
            }
            if (!ok) fail(abort_, a.err, 2);
            tc::mma_commit(bars + 8 * DONE);
            settle(bars + 8 * DONE, 0);
        }
    } else {
        if (!__all_sync(0xffffffffu, tc::mbar_wait(bars + 8 * DONE, 0, abort_))) {
            fail(abort_, a.err, 2);
        } else {
            tc::fence_after();
            const int row = warp * 32 + lane;
            const int ra = RA == 2 ? row >> 6 : 0, m = RA == 2 ? row & 63 : row, dq = m / CIN, ci = m % CIN;
            const bool valid = dq < 3 && !*abort_;
            for (int dx = dx0; dx < dx1; dx++)
                for (int t = 0; t < NB; t++) {
                    const int dr = ra - t + 2;
                    if (dr < 0 || dr > 2) continue;
                    const int tap = a.zring ? dr * 9 + dq * 3 + dx : dq * 9 + dr * 3 + dx;
                    for (int ch = 0; ch < COUT / 16; ch++) {
                        uint32_t rr[16];
                        tc::tmem_ld16(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(dx * N + t * COUT + ch * 16), rr);
                        tc::tmem_wait_ld();
                        if (valid)
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                atomicAdd(a.dw + ((size_t)tap * COUT + ch * 16 + j) * CIN + ci, __uint_as_float(rr[j]));
                        __syncwarp();
                    }
                }
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 8) tc::tmem_dealloc(tbase, NCOLS);
}

// ---- descriptor self-test ------------------------------------------------------------
// One CTA: A (128 x 32) and B (64 x 32) written by the threads into shared
// memory in a K-major or MN-major core-matrix layout, two MMAs (K = 16 each)
// into TMEM, the result compared with an exact FP32 product (all values are
// small multiples of 1/4, so every sum is exact).  Shared memory is sized so
// that every read stays inside it even if the LBO and SBO fields are swapped.
// swap = 2 issues no MMA: the completion wait then runs out after its time
// limit, which is how the bounded waits are tested (result: 1000000 + the
// wrong values of the untouched accumulator).
constexpr int ST_M = 128, ST_N = 64, ST_K = 32, ST_SMEM = 128 * 1024;

__device__ __forceinline__ float st_a(int m, int k) { return (float)(((m * 3 + k * 7) % 9) - 4) * 0.25f; }
__device__ __forceinline__ float st_b(int n, int k) { return (float)(((n * 5 + k * 3) % 7) - 3) * 0.5f; }

// mn = 2: both operands in the 128-byte-swizzle K-major layout (rows of 64
// elements, 16-byte chunk c of row r stored at chunk c ^ (r % 8)), K = 64 in
// four MMAs advancing 32 bytes; A starts `swap` (0..7) rows into a 136-row
// tile.  The swizzle is applied to absolute shared-memory address bits, so a
// start that is not 1024-byte aligned needs no base offset (field left 0).
// mn = 3: both operands in the 128-byte-swizzle MN-major layout (rows of 64 M
// or N elements, one per K), A of two atoms starting `swap` K rows in.
constexpr int SW_K = 64;
__device__ __forceinline__ float sw_a(int p, int k) { return (float)(((p * 5 + k * 3) % 11) - 5) * 0.25f; }

__global__ void __launch_bounds__(128) k_umma_selftest(int mn, int swap, unsigned long long *bad)
{
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t bar[1];
    __shared__ uint32_t tslot;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s0 = (tc::smem_u32(dsm) + 1023u) & ~1023u;
    uint8_t *g0 = dsm + (s0 - tc::smem_u32(dsm));
    const uint32_t offB = 32 * 1024;
    if (threadIdx.x == 0) {
        abort_s = 0;
        tc::mbar_init(tc::smem_u32(bar), 1);
        tc::mbar_fence_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tc::smem_u32(&tslot), 64);
        tc::tmem_relinquish();
    }
    for (int i = threadIdx.x; i < (ST_SMEM - 1024) / 4; i += blockDim.x) reinterpret_cast<uint32_t *>(g0)[i] = 0u;
    __syncthreads();
    if (mn == 2) {
        for (int i = threadIdx.x; i < 136 * SW_K; i += blockDim.x) {
            int p = i / SW_K, k = i % SW_K;
            uint32_t off = (uint32_t)(p * 128 + (((k >> 3) ^ (p & 7)) << 4) + (k & 7) * 2);
            *reinterpret_cast<bf16 *>(g0 + off) = __float2bfloat16_rn(sw_a(p, k));
        }
        for (int i = threadIdx.x; i < ST_N * SW_K; i += blockDim.x) {
            int n = i / SW_K, k = i % SW_K;
            uint32_t off = (uint32_t)(n * 128 + (((k >> 3) ^ (n & 7)) << 4) + (k & 7) * 2);
            *reinterpret_cast<bf16 *>(g0 + offB + off) = __float2bfloat16_rn(st_b(n, k));
        }
    }
    if (mn == 3) {
        for (int i = threadIdx.x; i < 40 * ST_M; i += blockDim.x) {
            int p = i / ST_M, m = i % ST_M;
            uint32_t off = (uint32_t)((m >> 6) * 8192 + p * 128 + ((((m & 63) >> 3) ^ (p & 7)) << 4) + (m & 7) * 2);
            *reinterpret_cast<bf16 *>(g0 + off) = __float2bfloat16_rn(sw_a(p, m));
        }
        for (int i = threadIdx.x; i < ST_K * ST_N; i += blockDim.x) {
            int k = i / ST_N, n = i % ST_N;
            uint32_t off = (uint32_t)(k * 128 + (((n >> 3) ^ (k & 7)) << 4) + (n & 7) * 2);
            *reinterpret_cast<bf16 *>(g0 + offB + off) = __float2bfloat16_rn(st_b(n, k));
        }
    }
    for (int i = threadIdx.x; mn < 2 && i < ST_M * ST_K; i += blockDim.x) {
        int m = i / ST_K, k = i % ST_K;
        uint32_t off = mn ? (uint32_t)((m / 8) * (ST_K * 16) + (k / 8) * 128 + (k % 8) * 16 + (m % 8) * 2)
                          : (uint32_t)((k / 8) * (ST_M * 16) + (m / 8) * 128 + (m % 8) * 16 + (k % 8) * 2);
        *reinterpret_cast<bf16 *>(g0 + off) = __float2bfloat16_rn(st_a(m, k));
    }
    for (int i = threadIdx.x; mn < 2 && i < ST_N * ST_K; i += blockDim.x) {
        int n = i / ST_K, k = i % ST_K;
        uint32_t off = mn ? (uint32_t)((n / 8) * (ST_K * 16) + (k / 8) * 128 + (k % 8) * 16 + (n % 8) * 2)
                          : (uint32_t)((k / 8) * (ST_N * 16) + (n / 8) * 128 + (n % 8) * 16 + (k % 8) * 2);
        *reinterpret_cast<bf16 *>(g0 + offB + off) = __float2bfloat16_rn(st_b(n, k));
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tbase = tslot;
    if (threadIdx.x == 0 && mn == 2) {
        uint32_t idesc = tc::idesc_bf16(ST_M, ST_N, 0, 0);
        uint32_t sh = (uint32_t)swap & 7u;
        for (int ks = 0; ks < SW_K / 16; ks++) {
            uint32_t aa = s0 + sh * 128u + (uint32_t)ks * 32u, bb = s0 + offB + (uint32_t)ks * 32u;
            uint64_t ad = tc::sdesc(aa, 16, 1024) | (2ull << 61);
            uint64_t bd = tc::sdesc(bb, 16, 1024) | (2ull << 61);
            tc::mma_bf16(tbase, ad, bd, idesc, ks > 0);
        }
        tc::mma_commit(tc::smem_u32(bar));
    } else if (threadIdx.x == 0 && mn == 3) {
        uint32_t idesc = tc::idesc_bf16(ST_M, ST_N, 1, 1);
        for (int ks = 0; ks < ST_K / 16; ks++)
            tc::mma_bf16(tbase, mn128_desc(s0 + ((uint32_t)swap & 7u) * 128u + (uint32_t)ks * 2048u, 8192u),
                         mn128_desc(s0 + offB + (uint32_t)ks * 2048u, 8192u), idesc, ks > 0);
        tc::mma_commit(tc::smem_u32(bar));
    } else if (threadIdx.x == 0 && swap != 2) {
        // (K-group stride, M/N-group stride) of the layouts written above
        uint32_t a_k = mn ? 128u : ST_M * 16u, a_m = mn ? ST_K * 16u : 128u;
        uint32_t b_k = mn ? 128u : ST_N * 16u, b_n = mn ? ST_K * 16u : 128u;
        uint32_t idesc = tc::idesc_bf16(ST_M, ST_N, mn, mn);
        for (int ks = 0; ks < ST_K / 16; ks++) {
            uint32_t aa = s0 + (uint32_t)ks * 2u * a_k, bb = s0 + offB + (uint32_t)ks * 2u * b_k;
            uint64_t ad = swap ? tc::sdesc(aa, a_m, a_k) : tc::sdesc(aa, a_k, a_m);
            uint64_t bd = swap ? tc::sdesc(bb, b_n, b_k) : tc::sdesc(bb, b_k, b_n);
            tc::mma_bf16(tbase, ad, bd, idesc, ks > 0);
        }
        tc::mma_commit(tc::smem_u32(bar));
    }
    bool ok = tc::mbar_wait(tc::smem_u32(bar), 0, &abort_s);
    tc::fence_after();
    unsigned long long nbad = ok ? 0ull : 1000000ull;
    int row = (warp & 3) * 32 + lane;
    for (int ch = 0; ch < ST_N / 16; ch++) {
        uint32_t rr[16];
        tc::tmem_ld16(tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)ch * 16u, rr);
        tc::tmem_wait_ld();
        for (int j = 0; j < 16; j++) {
            int n = ch * 16 + j;
            float ref = 0.f;
            if (mn == 2) {
                for (int k = 0; k < SW_K; k++) ref += sw_a(row + (swap & 7), k) * st_b(n, k);
            } else if (mn == 3) {
                for (int k = 0; k < ST_K; k++) ref += sw_a(k + (swap & 7), row) * st_b(n, k);
            } else {
                for (int k = 0; k < ST_K; k++) ref += st_a(row, k) * st_b(n, k);
            }
            if (__uint_as_float(rr[j]) != ref) nbad++;
        }
    }
    atomicAdd(bad, nbad);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0) tc::tmem_dealloc(tbase, 64);
}

// ---- weight packing ------------------------------------------------------------------
// K elements k of a tap's B operand (rows n of 128 bytes, 128-byte swizzled:
// 16-byte chunk c of row n at chunk c ^ (n % 8)); W[tap][n][k] forward,
// W[26 - tap][k][n] for the data gradient.
// k_conv_wide, per (channel chunk of kc, tap): row n holds k = 0 .. kc-1.
// k_conv_rows, per (dx, block of 64 K): row dr * N + n, K = dq * cin + k with
// (r, q) = (y, z) or, zring, (z, y).
__device__ __forceinline__ long long pack_index(const ConvPlan &p, int kin, int nout, int tap, int n, int k)
{
    long long row;
    int k64;
    if (p.rows) {
        const int dx = tap % 3, dy = (tap / 3) % 3, dz = tap / 9;
        const int K = (p.zring ? dy : dz) * kin + k;
        row = (long long)(dx * rows_nkb(kin) + (K >> 6)) * (3 * nout) + (p.zring ? dz : dy) * nout + n;
        k64 = K & 63;
    } else {
        const int kci = k / p.kc;
        row = (long long)(kci * 27 + tap) * nout + n;
        k64 = k - kci * p.kc;
    }
    return row * 64 + (((k64 >> 3) ^ ((int)row & 7)) << 3) + (k64 & 7);
}

__global__ void k_pack(const float *__restrict__ W, int cin, int cout, ConvPlan pf, ConvPlan pb, bf16 *__restrict__ wf,
                       bf16 *__restrict__ wd)
{
    long long n = 27LL * cin * cout;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        int ci = (int)(idx % cin);
        long long t = idx / cin;
        int co = (int)(t % cout), tap = (int)(t / cout);
        bf16 w = __float2bfloat16_rn(W[idx]);
        wf[pack_index(pf, cin, cout, tap, co, ci)] = w;
        wd[pack_index(pb, cout, cin, 26 - tap, ci, co)] = w;
    }
}

// ---- host -----------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

int get_encode()
{
    std::call_once(g_encode_once, []() {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    return g_encode ? 0 : 1;
}

// channel-blocked tensor [C/8][Z][Y][X][8] as a 5-D map (8, X, Y, Z, C/8)
int make_map(CUtensorMap *m, const void *ptr, int X, int Y, int Z, int C, int b1, int b2, int b3, int b4)
{
    if (get_encode()) { snprintf(g_conv_err, sizeof(g_conv_err), "cuTensorMapEncodeTiled unavailable"); return 1; }
    cuuint64_t dims[5] = {8, (cuuint64_t)X, (cuuint64_t)Y, (cuuint64_t)Z, (cuuint64_t)(C / 8)};
    cuuint64_t str[4] = {16, (cuuint64_t)X * 16, (cuuint64_t)X * Y * 16, (cuuint64_t)X * Y * Z * 16};
    cuuint32_t box[5] = {8, (cuuint32_t)b1, (cuuint32_t)b2, (cuuint32_t)b3, (cuuint32_t)b4};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(ptr), dims, str, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(g_conv_err, sizeof(g_conv_err), "cuTensorMapEncodeTiled failed (%d) for %dx%dx%dx%d box %d,%d,%d,%d",
                 (int)r, X, Y, Z, C, b1, b2, b3, b4);
        return 1;
    }
    return 0;
}

inline uint32_t r1024(uint32_t v) { return (v + 1023u) & ~1023u; }

void tile_dims(int X, int Y, int Z, int &bx, int &by, int &bz)
{
    bx = X < 128 ? X : 128;
    by = Y < 128 / bx ? Y : 128 / bx;
    bz = Z < 128 / (bx * by) ? Z : 128 / (bx * by);
}

// largest dynamic shared memory a launch of fn may request (opt-in limit
// minus the kernel's static shared memory); set as fn's attribute once
int dyn_smem_limit(const void *fn)
{
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return 0;
    int lim = optin - (int)fa.sharedSizeBytes;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess) return 0;
    return lim;
}

int launch_error(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return 0;
    snprintf(g_conv_err, sizeof(g_conv_err), "%s launch: %s", what, cudaGetErrorString(e));
    return 1;
}

// resident CTAs per SM allowed by shared memory (228 KB per SM, 1 KB reserved
// per CTA) and TMEM (512 columns), at most 4
int ctas_per_sm(uint32_t smem, int ncols)
{
    int n = (int)((228u * 1024u) / (smem + 1024u + 512u));
    int t = 512 / ncols;
    if (n > t) n = t;
    if (n > 4) n = 4;
    return n < 1 ? 1 : n;
}


}  // namespace

const char *conv_last_error() { return g_conv_err; }

ConvPlan conv_plan(int X, int Y, int Z, int cin, int cout)
{
    ConvPlan p{};
    p.rows = cin <= 32 && cout <= 32;
    p.zring = X < 128;
    const int most = X < 128 ? 64 : 32;
    p.kc = cin < most ? cin : most;
    return p;
}

void conv_pack_weights(cudaStream_t s, const float *W, int cin, int cout, const ConvPlan &pf, const ConvPlan &pb,
                       bf16 *wf, bf16 *wd)
{
    long long n = 27LL * cin * cout;
    int nb = (int)((n + 255) / 256);
    k_pack<<<nb < 2048 ? nb : 2048, 256, 0, s>>>(W, cin, cout, pf, pb, wf, wd);
}

namespace {

template <int CIN, int COUT, int ZRING>
int launch_rows(cudaStream_t s, RowArgs r, int nsm, int pdl)
{
    constexpr uint32_t smem = rows_smem(CIN, COUT);
    static int lim = dyn_smem_limit((const void *)k_conv_rows<CIN, COUT, ZRING>);
    if ((int)smem > lim) { snprintf(g_conv_err, sizeof(g_conv_err), "conv rows needs %u B of shared memory", smem); return 1; }
    const int most = nsm * ctas_per_sm(smem, NBLK * COUT);
    // an item of rch costs rch + 2 inputs: up to 32, fewer where that leaves
    // CTAs without two items; below 4 only where CTAs would have none
    const long long lines = (long long)r.ntx * r.R;
    r.rch = 32;
    while ((r.rch > 4 && lines / r.rch < 2LL * most) || (r.rch > 1 && lines / r.rch < most)) r.rch >>= 1;
    r.nitems = r.ntx * ((r.R + r.rch - 1) / r.rch);
    net_launch(pdl, k_conv_rows<CIN, COUT, ZRING>, most < r.nitems ? most : r.nitems, 1, 288, smem, s, r);
    return launch_error("k_conv_rows");
}

template <int ZRING>
int launch_rows(cudaStream_t s, const RowArgs &r, int cin, int cout, int nsm, int pdl)
{
    if (cin == 16) return cout == 16 ? launch_rows<16, 16, ZRING>(s, r, nsm, pdl) : launch_rows<16, 32, ZRING>(s, r, nsm, pdl);
    return cout == 16 ? launch_rows<32, 16, ZRING>(s, r, nsm, pdl) : launch_rows<32, 32, ZRING>(s, r, nsm, pdl);
}

}  // namespace

int conv3_fwd(cudaStream_t s, const bf16 *in, int X, int Y, int Z, int cin, int cout, const bf16 *wpk,
              const ConvEpi &e, int *err, int nsm, int pdl)
{
    if (cin % 16 || cout % 16 || cout > 128 || cin > 128) { snprintf(g_conv_err, sizeof(g_conv_err), "conv channels"); return 1; }
    const ConvPlan p = conv_plan(X, Y, Z, cin, cout);
    const EpiP epi{e.bias, e.relu, e.mask, e.out, e.headw, e.headb, e.hout, (size_t)X * Y * Z};
    if (p.rows) {
        RowArgs r{};
        r.X = X;
        r.W = X % 128 ? X + 2 : X;
        r.R = p.zring ? Z : Y; r.rs = p.zring ? X * Y : X;
        r.Q = p.zring ? Y : Z; r.qs = p.zring ? X : X * Y;
        r.ntx = (int)(((long long)r.Q * r.W + 127) / 128);
        r.in = in; r.wpk = wpk; r.epi = epi; r.err = err;
        return p.zring ? launch_rows<1>(s, r, cin, cout, nsm, pdl) : launch_rows<0>(s, r, cin, cout, nsm, pdl);
    }
    WideArgs a{};
    a.X = X; a.Y = Y; a.Z = Z; a.W = X + 2;
    a.cin = cin; a.cout = cout; a.kc = p.kc; a.nkc = (cin + p.kc - 1) / p.kc;
    a.ntiles = (int)(((long long)Z * Y * a.W + 127) / 128);
    // output channels per CTA: halved while that still gives every CTA an SM of its own
    a.nt = cout;
    while (a.nt % 32 == 0 && (long long)a.ntiles * (cout / a.nt) * 2 <= nsm) a.nt >>= 1;
    a.nsplit = cout / a.nt;
    a.stride = SBYTES + 3u * (uint32_t)a.nt * 128u;
    a.in = in; a.wpk = wpk; a.epi = epi; a.err = err;
    static int lim = dyn_smem_limit((const void *)k_conv_wide);
    a.stages = (lim - 1024) / (int)a.stride;
    if (a.stages > WSTAGES) a.stages = WSTAGES;
    if (a.stages <= WLAG) { snprintf(g_conv_err, sizeof(g_conv_err), "conv needs %u B of shared memory a stage", a.stride); return 1; }
    const int nwork = a.ntiles * a.nsplit;
    net_launch(pdl, k_conv_wide, nsm < nwork ? nsm : nwork, 1, 288, (uint32_t)a.stages * a.stride + 1024u, s, a);
    return launch_error("k_conv_wide");
}

namespace {

template <int CIN, int COUT>
int launch_wgrad_rows(cudaStream_t s, WgRowArgs r, int nsm, int pdl)
{
    constexpr uint32_t smem = WRS * wgr_stage(CIN, COUT) + 1024u;
    static int lim = dyn_smem_limit((const void *)k_wgrad_rows<CIN, COUT>);
    if ((int)smem > lim) { snprintf(g_conv_err, sizeof(g_conv_err), "wgrad needs %u B of shared memory", smem); return 1; }
    r.nsteps = r.ntx * ((r.R + WgR<CIN>::RA - 1) / WgR<CIN>::RA);
    r.ndx = r.nsteps > 20 * nsm ? 1 : 3;
    const int ng = 3 / r.ndx, per = nsm / ng < r.nsteps ? nsm / ng : r.nsteps;
    net_launch(pdl, k_wgrad_rows<CIN, COUT>, ng * (per > 0 ? per : 1), 1, 288, smem, s, r);
    return launch_error("k_wgrad_rows");
}

}  // namespace

int conv3_wgrad(cudaStream_t s, const bf16 *x, const bf16 *dy, int X, int Y, int Z, int cin, int cout, float *dw,
                int *err, int nsm, int pdl)
{
    if (cin % 16 || cout % 16 || cout > 128 || cin > 128) { snprintf(g_conv_err, sizeof(g_conv_err), "wgrad channels"); return 1; }
    WgArgs a{};
    tile_dims(X, Y, Z, a.bx, a.by, a.bz);
    a.nb = a.bx * a.by * a.bz;
    if (a.nb % 16) {   // of k_wgrad; a grid is taken or refused whichever kernel its channels choose
        snprintf(g_conv_err, sizeof(g_conv_err), "wgrad voxel tile %dx%dx%d is no multiple of 16", a.bx, a.by, a.bz);
        return 1;
    }
    if (cin <= 32 && cout <= 32) {
        WgRowArgs r{};
        r.zring = X < 128;
        r.X = X;
        r.W = X % 128 ? X + 2 : X;
        r.R = r.zring ? Z : Y; r.rs = r.zring ? X * Y : X;
        r.Q = r.zring ? Y : Z; r.qs = r.zring ? X : X * Y;
        r.cstep = X * Y * Z;
        r.ntx = (int)(((long long)r.Q * r.W + 127) / 128);
        r.x = x; r.dy = dy; r.dw = dw; r.err = err;
        if (cin == 16) return cout == 16 ? launch_wgrad_rows<16, 16>(s, r, nsm, pdl) : launch_wgrad_rows<16, 32>(s, r, nsm, pdl);
        return cout == 16 ? launch_wgrad_rows<32, 16>(s, r, nsm, pdl) : launch_wgrad_rows<32, 32>(s, r, nsm, pdl);
    }
    a.X = X; a.Y = Y; a.Z = Z; a.cin = cin; a.cout = cout;
    a.G = 128 / cin; a.ngroups = (27 + a.G - 1) / a.G;
    a.ntx = (X + a.bx - 1) / a.bx; a.nty = (Y + a.by - 1) / a.by; a.ntz = (Z + a.bz - 1) / a.bz;
    a.ntiles = a.ntx * a.nty * a.ntz;
    a.tapbytes = (uint32_t)a.nb * cin * 2u;
    a.bbytes = (uint32_t)a.nb * cout * 2u;
    // operand reads span 128 rows per 8 channels: keep that much room per stage
    uint32_t abig = 128u * 16u * (uint32_t)(a.G * cin / 8), bbig = 128u * 16u * (uint32_t)(cout / 8);
    uint32_t aroom = (uint32_t)a.G * a.tapbytes;
    a.stride = r1024((aroom > abig ? aroom : abig) + (a.bbytes > bbig ? a.bbytes : bbig));
    uint32_t smem = WG_STAGES * a.stride + 1024u;
    CUtensorMap mx, md;
    if (make_map(&mx, x, X, Y, Z, cin, a.bx, a.by, a.bz, cin / 8)) return 1;
    if (make_map(&md, dy, X, Y, Z, cout, a.bx, a.by, a.bz, cout / 8)) return 1;
    static int lim = dyn_smem_limit((const void *)k_wgrad);
    if ((int)smem > lim) { snprintf(g_conv_err, sizeof(g_conv_err), "wgrad needs %u B of shared memory", smem); return 1; }
    int want = 2 * nsm / a.ngroups;
    a.nsplit = want < 1 ? 1 : want;
    if (a.nsplit > a.ntiles) a.nsplit = a.ntiles;
    a.dw = dw; a.err = err;
    net_launch(pdl, k_wgrad, a.ngroups * a.nsplit, 1, 192, smem, s, mx, md, a);
    return launch_error("k_wgrad");
}

int conv_selftest_umma(int mn_major, int swap, unsigned long long *mismatches)
{
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(*d));
    cudaFuncSetAttribute(k_umma_selftest, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM);
    k_umma_selftest<<<1, 128, ST_SMEM>>>(mn_major, swap, d);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) { snprintf(g_conv_err, sizeof(g_conv_err), "%s", cudaGetErrorString(e)); return 1; }
    return 0;
}
