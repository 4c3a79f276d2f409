// turb_mg.cuh -- multigrid hierarchy descriptors (device pointers).
#pragma once
#include <cuda.h>

#include <vector>

#include "turb_internal.cuh"

#define TURB_MG_MAXLEV 24
#define MG_TAIL_MAXLEV 6   // levels a fused single-block V-cycle tail may hold
#define MG_CLUSTER_MAXLEV 8   // levels a one-cluster V-cycle launch may hold
// the shared-memory V-cycle of the lower levels (k_mglow.cu): levels it may
// hold, cells of the level it starts from by default (FP32, FP64), cells up
// to which a level is swept by one block, cells of a coarsest level whose
// inverse is staged, and the most shared memory a block may take
#define MG_LOW_MAXLEV 8
#define MG_LOW_CELLS32 32768
#define MG_LOW_CELLS64 32768
#define MG_LOW_ONE32 4096
#define MG_LOW_ONE64 512
#define MG_LOW_INV 64
#define MG_LOW_SMEM (220 * 1024)   // beside 4 KB of static shared memory

// 1-D transfer tables between a level and the next coarser one along one
// direction: prolongation weights per fine index (two coarse cells) and the
// transposed (restriction) lists per coarse index (up to four fine cells).
struct Xfer1D {
    const int *I0, *I1;
    const double *w0d, *w1d;
    const float *w0f, *w1f;
    const int *rcnt, *rf;
    const double *rwd;
    const float *rwf;
};

// the host's copy of the tables of one direction
struct MgXferHost {
    std::vector<int> I0, I1, rf;
    std::vector<double> w0, w1, rw;
};

struct MgDevLevel {
    int nx, ny, nz;
    int cx, cy, cz;                                   // coarsened into next level
    Xfer1D tx, ty, tz;                                // transfer to the next level
    const double *dxd, *dyd, *dzd, *rfxd, *rfyd, *rfzd;
    const float *dxf, *dyf, *dzf, *rfxf, *rfyf, *rfzf;
    // the x tables split by parity for 4-cell float4 reads (nx even): entry
    // par * nx/2 + m is cell i = 2m + par: dx[i], 1/f of its left face
    // (rfx[i]) and of its right face (rfx[i+1])
    const float *dxpf = nullptr, *rlpf = nullptr, *rrpf = nullptr;
    // the 1-D tables packed for k_vcycle_low (mg_low_tables), FP32 and FP64
    const unsigned char *lowf = nullptr, *lowd = nullptr;
    double pin;
    // colour-split storage (x, b, invd; not r): with nx even, cell c of colour
    // (i+j+k)&1 lives at colour*(n/2) + c/2, so a red-black half sweep reads
    // and writes dense half arrays
    int split = 0;
};

// the finest FP32 level's two-sweeps-per-pass smoother (k_rbtb.cu): TMA
// maps of x (both ping-pong arrays), b and 1/diag, and the launch shape
struct RbTbPlan {
    CUtensorMap mx[2];
    MgDevLevel lev;
    const float *b = nullptr, *invd = nullptr;
    float *xo[2];
    int tiles_x = 0, ntiles = 0, grid = 0;
    int *err = nullptr;
    int ok = 0;
};
int mg_tb_plan(RbTbPlan *p, const MgDevLevel &L0, float *x0, float *x1, const float *b0, const float *invd0, int *err);
void mg_tb_sweeps(cudaStream_t s, const RbTbPlan &p, int in, int c0, int zero_init, int pdl);
size_t mg_tb_smem();

template <typename T>
struct MgHier {
    int nl;
    MgDevLevel lev[TURB_MG_MAXLEV];
    T *x[TURB_MG_MAXLEV], *b[TURB_MG_MAXLEV], *r[TURB_MG_MAXLEV], *invd[TURB_MG_MAXLEV];
    const double *coarse_inv;
    // from this level on (-1: never) the V-cycle runs as one launch: of one
    // cluster with x in shared memory (k_vcycle_low) where mg_low_fits, else
    // of a single block (k_vcycle_tail, at most MG_TAIL_MAXLEV levels)
    int tail_from = -1;
    int low_ctas = 0;   // blocks of k_vcycle_low's cluster (mg_low_ctas; 0: not used)
    // 1: FP32 half sweeps after the first of a cycle march along k (k_rbgs4z)
    int marching = 0;
    // 1: FP64 half sweeps and residuals of large levels march along k
    // (k_rbgs_col, k_resid_col); 0: k_rbgs, k_resid throughout
    int columns = 1;
    int nsm = 1;   // SMs of the device
    // 1: the kernels of the V-cycle and of the CG step use programmatic dependent launch
    int pdl = 1;
    // from this level on (-1: never) the V-cycle runs as one launch of one
    // thread-block cluster of cluster_ctas blocks (k_vcycle_cluster)
    int cluster_from = -1;
    int cluster_ctas = 0;
    // level 0 (FP32 only): pairs of sweeps in one pass each (k_rbgs_tb), when set
    const RbTbPlan *tb = nullptr;
};

template <typename T>
void mg_setup_invdiag(cudaStream_t s, const MgDevLevel &L, T *invd);
template <typename T>
// level l smooths with pre[l] / post[l] red-black sweeps
void mg_vcycle(cudaStream_t s, const MgHier<T> &H, int l, const int *pre, const int *post);
int mg_vcycle_launches(int nl, const int *pre, const int *post, int tail_from, int cluster_from = -1, int tb0 = 0);
template <typename T>
int mg_cluster_ctas();
// the shared-memory V-cycle of level l and below (k_mglow.cu): mg_low launches
// it and returns 1, or returns 0 where those levels do not fit
template <typename T>
int mg_low_ctas();
// a level's 1-D tables packed for it: widths, 1/face distances and the
// transfer tables to the next level, each along x, y, z
template <typename T>
std::vector<unsigned char> mg_low_tables(const MgDevLevel &F, const MgDevLevel &C, const std::vector<T> (&dd)[3],
                                         const std::vector<T> (&rf)[3], const MgXferHost (&x)[3]);
template <typename T>
int mg_low_fits(const MgHier<T> &H, int l);
template <typename T>
int mg_low(cudaStream_t s, const MgHier<T> &H, int l, const int *pre, const int *post);
template <typename T>
double mg_vcycle_bytes(const MgHier<T> &H, int l, const int *pre, const int *post);

// Linear prolongation of the eight coarse values around a cell (x fastest,
// then y, z; w*0, w*1 the weights of the lower and upper one), summed in that
// order with every rounding explicit, so that every kernel gives the same
// bits (an absent neighbour has weight 0 and the value of its pair)
__device__ __forceinline__ float mg_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mg_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mg_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mg_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename T>
__device__ __forceinline__ T mg_prolong8(const T (&v)[8], T wx0, T wx1, T wy0, T wy1, T wz0, T wz1)
{
    T acc = 0;
#pragma unroll
    for (int e = 0; e < 8; e++)
        acc = mg_fma(mg_mul(mg_mul(e & 4 ? wz1 : wz0, e & 2 ? wy1 : wy0), e & 1 ? wx1 : wx0), v[e], acc);
    return acc;
}
// the 4 x 4 entries of one plane of a restriction (weights wz * wy[d] *
// wx[f]) added to s, in that order; cx 0: x is not coarsened, entry f = 0 of
// weight 1 alone
template <typename T>
__device__ __forceinline__ T mg_restrict16(T s, const T (&v)[4][4], T wz, const T *wy, const T *wx, bool cx)
{
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const T w = mg_mul(wz, wy[d]);
        if (cx) {
#pragma unroll
            for (int f = 0; f < 4; f++) s = mg_fma(mg_mul(w, wx[f]), v[d][f], s);
        } else {
            s = mg_fma(w, v[d][0], s);
        }
    }
    return s;
}

// FP64 CG vector kernels on the compact level-0 layout (k_pcg.cu)
struct PcgScal {
    double bb, rr, rz, zr_old, rz_old, pq, alpha, beta;   // slot order is used by the reductions
};
void pcg_gather(cudaStream_t s, const Dims &d, const MgDevLevel &L0, const double *phi_da, const double *pb_da,
                double *x, double *bw);
void pcg_scatter(cudaStream_t s, const Dims &d, const MgDevLevel &L0, const double *x, double *phi_da);
// The sums of these end in the launch itself (the last block adds the
// partials; count: a zero word the launch leaves zero): |r|^2, p.q and alpha,
// a.b, r.z, z.r_old and beta, |r|^2 (also to the page-locked *host_rr).  With
// count null, pcg_resid and pcg_apply leave the partials for pcg_reduce.  pdl:
// the kernel may be scheduled while the one ahead of it drains
void pcg_resid(cudaStream_t s, const MgDevLevel &L0, const double *bw, const double *x, double *r, double *part,
               double *dst, unsigned *count);
void pcg_apply(cudaStream_t s, const MgDevLevel &L0, const double *p, double *q, double *part, PcgScal *sc,
               unsigned *count, int pdl);
void pcg_dot(cudaStream_t s, long long n, const double *a, const double *b, double *part, double *dst, unsigned *count);
void pcg_dot2(cudaStream_t s, long long n, const double *r, const double *z, const double *rold, double *part,
              PcgScal *sc, int restart, unsigned *count, int pdl);
int pcg_stencil_parts(const MgDevLevel &L);
void pcg_reduce(cudaStream_t s, const double *part, int nvals, double *dst, int nper = 0);
void pcg_pupdate(cudaStream_t s, long long n, const double *z, double *p, const PcgScal *sc, int first, int pdl);
void pcg_xrupdate(cudaStream_t s, long long n, double *x, double *r, double *rold, const double *p,
                  const double *q, PcgScal *sc, double *part, double *host_rr, unsigned *count, int pdl);
void pcg_to_float(cudaStream_t s, long long n, const double *a, float *b);
void pcg_to_double(cudaStream_t s, long long n, const float *a, double *b);
// the same into / out of a level's storage order (colour-split or not)
void mg_to_float(cudaStream_t s, const MgDevLevel &L, const double *a, float *b);
void mg_to_double(cudaStream_t s, const MgDevLevel &L, const float *a, double *b, int pdl = 0);
void pcg_copy(cudaStream_t s, long long n, const double *a, double *b);
int pcg_nparts();
void pcg_lincomb(cudaStream_t s, long long n, double a, const double *x, double b, const double *y, double *out);

// Galerkin fit of the initial guess (k_pcg.cu): up to GAL_MAX candidate
// solutions y_m, each with w_m = the right-hand side it solved (resid 0) or
// its computed residual (resid 1)
#define GAL_MAX 3
struct GalDirs {
    const double *y[GAL_MAX];
    const double *w[GAL_MAX];
    int resid[GAL_MAX];
    int nd;
};
struct GalCoef {
    double a[GAL_MAX];
};
// dst[a * GAL_MAX + b] = d_a . s_b, dst[GAL_MAX^2 + a] = d_a . r1 (part: >= 12 * 512 doubles)
void pcg_gal_dots(cudaStream_t s, long long n, const GalDirs &dd, const double *x0, const double *r1,
                  const double *bw, double *part, double *dst);
void pcg_gal_update(cudaStream_t s, long long n, const GalDirs &dd, const GalCoef &al, const double *x0, double *x);
// *dst = max_c |r_c| / (dx dy dz)_c on level 0 (part: >= pcg_stencil_parts(L0) doubles)
void pcg_rmax(cudaStream_t s, const MgDevLevel &L0, const double *r, double *part, double *dst);
