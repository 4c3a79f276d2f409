// k_pcg.cu -- FP64 conjugate-gradient vector kernels for the pressure solve
// (volume-weighted system on the compact physical-cell layout).  Dot products
// reduce into a fixed set of per-block partials that the block which finishes
// last sums in a fixed order, so results are run-to-run deterministic.
#include <algorithm>

#include "turb_internal.cuh"
#include "turb_mg.cuh"
#include "turb_sum.cuh"

namespace {

constexpr int NP = 4096;   // blocks of the grid-stride reductions
constexpr int BS = 256;
constexpr int VB = 4;      // blocks of a reduction that a block of its launch stands for

__device__ __forceinline__ void block_store(double v, double *dst)
{
    __shared__ double sm[32];
    int lt = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    v = warp_sum(v);
    if ((lt & 31) == 0) sm[lt >> 5] = v;
    __syncthreads();
    if (lt < 32) {
        double r = (lt < (nt >> 5)) ? sm[lt] : 0.0;
        r = warp_sum(r);
        if (lt == 0) *dst = r;
    }
    __syncthreads();
}

// block_store of NV values of a 256-thread block to dst + n * stride
template <int NV>
__device__ __forceinline__ void block_store256(const double (&v)[NV], double *dst, long long stride)
{
    double s[NV];
    block_sum256<NV>(v, s);
    if (threadIdx.x == 0 && threadIdx.y == 0)
#pragma unroll
        for (int n = 0; n < NV; n++) dst[n * stride] = s[n];
}

constexpr int KC = 4;   // planes per thread in the 3-D stencil kernels
__device__ __forceinline__ long long blk3() { return ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x; }

// (S x)_c = dz_k [cxy x_c - sum_xy a_n x_n] + (dx dy) [zs x_c - zb x_b - zf x_f]
// (+ the corner pin): the x and y face coefficients times the other cell
// widths are constants of the thread's (i, j) column and are formed once,
// the z ones are constants of a plane; absent faces have a zero coefficient
// (their neighbour index is redirected to the cell itself).  Eleven FP64
// operations per cell.
struct SCol {
    double axw, axe, ays, ayn, cxy, wz;
};

__device__ __forceinline__ SCol s_col(const MgDevLevel &L, int i, int j)
{
    SCol r;
    double dx = L.dxd[i], dy = L.dyd[j];
    double fxw = i > 0 ? L.rfxd[i] : 0.0, fxe = i < L.nx - 1 ? L.rfxd[i + 1] : 0.0;
    double fys = j > 0 ? L.rfyd[j] : 0.0, fyn = j < L.ny - 1 ? L.rfyd[j + 1] : 0.0;
    r.axw = dy * fxw;
    r.axe = dy * fxe;
    r.ays = dx * fys;
    r.ayn = dx * fyn;
    r.cxy = (r.axw + r.axe) + (r.ays + r.ayn);
    r.wz = dx * dy;
    return r;
}

// z face coefficients of one plane (zero for an absent face) and their sum
struct SPlane {
    double zb, zf, zs, dz;
};

__device__ __forceinline__ SPlane s_plane(const MgDevLevel &L, int k)
{
    SPlane r;
    r.zb = k > 0 ? L.rfzd[k] : 0.0;
    r.zf = k < L.nz - 1 ? L.rfzd[k + 1] : 0.0;
    r.zs = r.zb + r.zf;
    r.dz = L.dzd[k];
    return r;
}

// the n planes of a block from k0, formed once by its first threads
__device__ __forceinline__ void s_planes(const MgDevLevel &L, SPlane *sp, int k0, int n)
{
    int t = threadIdx.y * blockDim.x + threadIdx.x, k = k0 + t;
    if (t < n && k < L.nz) sp[t] = s_plane(L, k);
    __syncthreads();
}

// f(group, c, x_c, (S x)_c) over the G groups of KC planes of the thread's
// column.  A block of G groups forms the column's coefficients (eight FP64
// operations) once for 4 G cells and reads the cells above and below as the
// march reaches them; each group's sum is stored apart, so the partials are
// those of blocks of one group.  x is not __restrict__: k_apply starts before
// the kernel that writes it has ended.
template <int G, typename F>
__device__ __forceinline__ void s_march(const MgDevLevel &L, const double *x, F f)
{
    __shared__ SPlane sp[KC * G];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k0 = blockIdx.z * KC * G;
    s_planes(L, sp, k0, KC * G);
    if (i >= L.nx || j >= L.ny) return;
    const SCol a = s_col(L, i, j);
    const long long nx = L.nx, nxy = nx * L.ny;
    const long long ow = i > 0 ? 1 : 0, oe = i < L.nx - 1 ? 1 : 0, os = j > 0 ? nx : 0, on = j < L.ny - 1 ? nx : 0;
    const bool corner = i == L.nx - 1 && j == L.ny - 1;
    long long c = ((long long)k0 * L.ny + j) * nx + i;
    double xc = x[c], xb = k0 > 0 ? x[c - nxy] : xc;
#pragma unroll
    for (int g = 0; g < G; g++) {
#pragma unroll
        for (int kk = 0; kk < KC; kk++) {
            const int k = k0 + g * KC + kk;
            if (k >= L.nz) return;
            const SPlane z = sp[g * KC + kk];
            const double xf = k < L.nz - 1 ? x[c + nxy] : xc;
            const double xw = x[c - ow], xe = x[c + oe], xs = x[c - os], xn = x[c + on];
            double t = fma(a.axw, xw, fma(a.axe, xe, fma(a.ays, xs, a.ayn * xn)));
            double xy = fma(a.cxy, xc, -t);
            double sz = fma(z.zs, xc, -fma(z.zb, xb, z.zf * xf));
            double v = fma(z.dz, xy, a.wz * sz);
            if (corner && k == L.nz - 1) v = fma(L.pin, xc, v);
            f(g, c, xc, v);
            xb = xc;
            xc = xf;
            c += nxy;
        }
    }
}
// the G groups' sums to the partials of blocks of one group
template <int G>
__device__ __forceinline__ void store_groups(const MgDevLevel &L, const double (&acc)[G], double *part)
{
    double s[G];
    block_sum256<G>(acc, s);
    if (threadIdx.x == 0 && threadIdx.y == 0)
#pragma unroll
        for (int g = 0; g < G; g++) {
            const int b = blockIdx.z * G + g;
            if (b * KC < L.nz) part[((long long)b * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = s[g];
        }
}

__global__ void k_gather(Dims d, MgDevLevel L, const double *__restrict__ phi, const double *__restrict__ pb,
                         double *__restrict__ x, double *__restrict__ bw)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    if (i >= L.nx || j >= L.ny) return;
    long long c = ((long long)k * L.ny + j) * L.nx + i, p = d.at(i, j, k);
    x[c] = phi[p];
    bw[c] = (L.dxd[i] * L.dyd[j] * L.dzd[k]) * pb[p];
}

__global__ void k_scatter(Dims d, MgDevLevel L, const double *__restrict__ x, double *__restrict__ phi)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    if (i >= d.NX || j >= d.NY) return;
    long long p = d.at(i, j, k);
    phi[p] = (i < L.nx && j < L.ny && k < L.nz) ? x[((long long)k * L.ny + j) * L.nx + i] : 0.0;
}

// r = W b - S x with partial |r|^2 per group of planes
template <int G>
__global__ void k_resid(MgDevLevel L, const double *__restrict__ bw, const double *__restrict__ x,
                        double *__restrict__ r, double *__restrict__ part, int nparts, double *dst, unsigned *count)
{
    double acc[G] = {};
    s_march<G>(L, x, [&](int g, long long c, double, double sx) {
        double v = bw[c] - sx;
        r[c] = v;
        acc[g] += v * v;
    });
    store_groups<G>(L, acc, part);
    if (count && last_block(count, gridDim.x * gridDim.y * gridDim.z)) sum_parts<1>(part, 0, nparts, dst);
}

// The kernels of a CG step start before the one ahead of them has ended, so
// the vectors they read are not __restrict__: through such a pointer the
// compiler may load what that kernel is still writing before pdl_wait.

// q = S p with partial p.q per group of planes, then alpha = rz / p.q
template <int G>
__global__ void k_apply(MgDevLevel L, const double *p, double *q, double *part, int nparts, PcgScal *sc, unsigned *count)
{
    pdl_trigger();
    pdl_wait();
    double acc[G] = {};
    s_march<G>(L, p, [&](int g, long long c, double pc, double v) {
        q[c] = v;
        acc[g] += pc * v;
    });
    store_groups<G>(L, acc, part);
    if (count && last_block(count, gridDim.x * gridDim.y * gridDim.z)) {
        sum_parts<1>(part, 0, nparts, &sc->pq);
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            sc->alpha = sc->pq != 0.0 ? sc->rz / sc->pq : 0.0;
            sc->rz_old = sc->rz;
        }
    }
}

// The grid-stride reductions are those of NP blocks of BS threads (or as many
// as have elements); a block of a launch stands for VB of them, so that a
// thread has VB elements in flight and VB sums share the block's barriers.
// vb_first: the thread's first element in the u-th of them
__device__ __forceinline__ long long vb_first(int u) { return ((long long)blockIdx.x * VB + u) * BS + threadIdx.x; }
template <int NVAL>
__device__ __forceinline__ void store_vb(const double (&acc)[NVAL * VB], double *part, int nvb)
{
    double s[NVAL * VB];
    block_sum256<NVAL * VB>(acc, s);
    if (threadIdx.x == 0)
#pragma unroll
        for (int v = 0; v < NVAL; v++)
#pragma unroll
            for (int u = 0; u < VB; u++)
                if ((int)blockIdx.x * VB + u < nvb) part[(long long)v * NP + blockIdx.x * VB + u] = s[v * VB + u];
}

__global__ void k_dot(long long n, int nvb, const double *__restrict__ a, const double *__restrict__ b,
                      double *__restrict__ part, double *dst, unsigned *count)
{
    const long long stride = (long long)nvb * BS;
    double acc[VB] = {};
    for (long long o = 0; o < n; o += stride) {
        double av[VB], bv[VB];
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            const bool in = c < n && (int)blockIdx.x * VB + u < nvb;
            av[u] = in ? a[c] : 0.0;
            bv[u] = in ? b[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < VB; u++) acc[u] += av[u] * bv[u];
    }
    store_vb<1>(acc, part, nvb);
    if (last_block(count, gridDim.x)) sum_parts<1>(part, 0, nvb, dst);
}

// rz = r.z and zr_old = z.r_old, then beta (0 on a restart)
__global__ void __launch_bounds__(BS, 4) k_dot2(long long n, int nvb, const double *r, const double *z, const double *ro,
                                                   double *part, PcgScal *sc, int restart, unsigned *count)
{
    pdl_trigger();
    pdl_wait();
    const long long stride = (long long)nvb * BS;
    double acc[2 * VB] = {};
    for (long long o = 0; o < n; o += stride) {
        double zv[VB], rv[VB], ov[VB];
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            const bool in = c < n && (int)blockIdx.x * VB + u < nvb;
            zv[u] = in ? z[c] : 0.0;
            rv[u] = in ? r[c] : 0.0;
            ov[u] = in ? ro[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < VB; u++) {
            acc[u] += rv[u] * zv[u];
            acc[VB + u] += ov[u] * zv[u];
        }
    }
    store_vb<2>(acc, part, nvb);
    if (last_block(count, gridDim.x)) {
        sum_parts<2>(part, NP, nvb, &sc->rz);   // rz and, next to it, zr_old
        if (threadIdx.x == 0 && !restart) sc->beta = sc->rz_old != 0.0 ? (sc->rz - sc->zr_old) / sc->rz_old : 0.0;
    }
}

__global__ void k_reduce(const double *__restrict__ part, int nvals, int nper, double *__restrict__ dst)
{
    for (int v = 0; v < nvals; v++) {
        double acc = 0.0;
        for (int t = threadIdx.x; t < nper; t += blockDim.x) acc += part[(long long)v * nper + t];
        block_store(acc, dst + v);
    }
}

__global__ void k_pupdate(long long n, int nvb, const double *z, double *p, const PcgScal *sc, int first)
{
    pdl_trigger();
    pdl_wait();
    const double beta = first ? 0.0 : sc->beta;
    const long long stride = (long long)nvb * BS;
    for (long long o = 0; o < n; o += stride) {
        double zv[VB], pv[VB];
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            const bool in = c < n && (int)blockIdx.x * VB + u < nvb;
            zv[u] = in ? z[c] : 0.0;
            pv[u] = in && !first ? p[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            if (c < n && (int)blockIdx.x * VB + u < nvb) p[c] = first ? zv[u] : zv[u] + beta * pv[u];
        }
    }
}

// x += alpha p, r_old = r, r -= alpha q and |r|^2
__global__ void __launch_bounds__(BS, 3) k_xrupdate(long long n, int nvb, double *x, double *r, double *ro, const double *p,
                                                       const double *q, PcgScal *sc, double *part, double *host_rr,
                                                       unsigned *count)
{
    pdl_trigger();
    pdl_wait();
    const double alpha = sc->alpha;
    const long long stride = (long long)nvb * BS;
    double acc[VB] = {};
    for (long long o = 0; o < n; o += stride) {
        double rv[VB], xv[VB], pv[VB], qv[VB];
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            const bool in = c < n && (int)blockIdx.x * VB + u < nvb;
            rv[u] = in ? r[c] : 0.0;
            qv[u] = in ? q[c] : 0.0;
            xv[u] = in ? x[c] : 0.0;
            pv[u] = in ? p[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < VB; u++) {
            const long long c = vb_first(u) + o;
            if (c < n && (int)blockIdx.x * VB + u < nvb) {
                double rc = rv[u];
                ro[c] = rc;
                x[c] = xv[u] + alpha * pv[u];
                rc -= alpha * qv[u];
                r[c] = rc;
                acc[u] += rc * rc;
            }
        }
    }
    store_vb<1>(acc, part, nvb);
    if (last_block(count, gridDim.x)) {
        sum_parts<1>(part, 0, nvb, &sc->rr);
        if (threadIdx.x == 0) *host_rr = sc->rr;   // page-locked: the host reads it after its wait
    }
}

__global__ void k_lincomb(long long n, double a, const double *__restrict__ x, double b, const double *__restrict__ y,
                          double *__restrict__ out)
{
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        out[c] = a * x[c] + b * y[c];
}

__global__ void k_f2(long long n, const double *__restrict__ a, float *__restrict__ b)
{
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        b[c] = (float)a[c];
}
__global__ void k_d2(long long n, const float *__restrict__ a, double *__restrict__ b)
{
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        b[c] = (double)a[c];
}
__global__ void k_copy(long long n, const double *__restrict__ a, double *__restrict__ b)
{
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x)
        b[c] = a[c];
}

// Galerkin fit of the initial guess (projection onto earlier solutions):
// direction m is d_m = y_m - x0 with S-image s_m = w_m - bw + r1 when w_m is
// the right-hand side y_m was solved for (S y_m = w_m to that solve's
// tolerance), or s_m = r1 - w_m when w_m is the computed residual of a
// candidate y_m.  Per block: G[a][b] = d_a . s_b and g[a] = d_a . r1, value
// v = a * GAL_MAX + b (g at GAL_MAX * GAL_MAX + a) in part[v * GAL_NP + block].
constexpr int GAL_NP = 512;
__global__ void __launch_bounds__(BS) k_gal_dots(long long n, GalDirs dd, const double *__restrict__ x0,
                                                 const double *__restrict__ r1, const double *__restrict__ bw,
                                                 double *__restrict__ part)
{
    double G[GAL_MAX][GAL_MAX] = {}, gv[GAL_MAX] = {};
    const int nd = dd.nd;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        double xc = x0[c], rc = r1[c], sb = rc - bw[c];
        double d[GAL_MAX], sv[GAL_MAX];
#pragma unroll
        for (int m = 0; m < GAL_MAX; m++) {
            if (m < nd) {
                d[m] = dd.y[m][c] - xc;
                sv[m] = dd.resid[m] ? rc - dd.w[m][c] : dd.w[m][c] + sb;
            } else {
                d[m] = 0.0;
                sv[m] = 0.0;
            }
        }
#pragma unroll
        for (int a = 0; a < GAL_MAX; a++) {
            gv[a] = fma(d[a], rc, gv[a]);
#pragma unroll
            for (int b = 0; b < GAL_MAX; b++) G[a][b] = fma(d[a], sv[b], G[a][b]);
        }
    }
#pragma unroll
    for (int a = 0; a < GAL_MAX; a++) {
#pragma unroll
        for (int b = 0; b < GAL_MAX; b++)
            block_store256<1>({G[a][b]}, part + (long long)(a * GAL_MAX + b) * GAL_NP + blockIdx.x, 0);
        block_store256<1>({gv[a]}, part + (long long)(GAL_MAX * GAL_MAX + a) * GAL_NP + blockIdx.x, 0);
    }
}

// x = x0 + sum_m alpha_m (y_m - x0)
__global__ void k_gal_update(long long n, GalDirs dd, GalCoef al, const double *__restrict__ x0, double *__restrict__ x)
{
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        double xc = x0[c], v = xc;
        for (int m = 0; m < dd.nd; m++) v = fma(al.a[m], dd.y[m][c] - xc, v);
        x[c] = v;
    }
}

// largest |r_c| / (dx_i dy_j dz_k): the unweighted residual b - A phi of the
// volume-weighted system, whose maximum times dt is the largest divergence
// the projection with this phi leaves.  3-D launch as k_apply (KC planes per
// thread); 1/(dx dy) once per thread and 1/dz once per plane of a block, so a
// cell costs two multiplies.  Per block maxima into part (NaN kept).
__global__ void k_rmax(MgDevLevel L, const double *__restrict__ r, double *__restrict__ part)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    __shared__ double izs[KC];
    int t = threadIdx.y * blockDim.x + threadIdx.x;
    if (t < KC && blockIdx.z * KC + t < L.nz) izs[t] = 1.0 / L.dzd[blockIdx.z * KC + t];
    __syncthreads();
    double m = 0.0;
    if (i < L.nx && j < L.ny) {
        double ixy = 1.0 / (L.dxd[i] * L.dyd[j]);
        for (int kk = 0; kk < KC; kk++) {
            int k = blockIdx.z * KC + kk;
            if (k >= L.nz) break;
            long long c = ((long long)k * L.ny + j) * L.nx + i;
            m = turb_maxbits(m, fabs(r[c]) * ixy * izs[kk]);
        }
    }
    __shared__ double sm[32];
    int lt = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    m = turb_warp_maxbits(m);
    if ((lt & 31) == 0) sm[lt >> 5] = m;
    __syncthreads();
    if (lt < 32) {
        m = lt < (nt >> 5) ? sm[lt] : 0.0;
        m = turb_warp_maxbits(m);
        if (lt == 0) part[blk3()] = m;
    }
}

__global__ void k_max_parts(const double *__restrict__ part, int n, double *__restrict__ dst)
{
    double m = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) m = turb_maxbits(m, part[t]);
    __shared__ double sm[32];
    m = turb_warp_maxbits(m);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (int)(blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        m = turb_warp_maxbits(m);
        if (threadIdx.x == 0) *dst = m;
    }
}


}  // namespace


static unsigned nblk(long long n);

void pcg_gal_dots(cudaStream_t s, long long n, const GalDirs &dd, const double *x0, const double *r1,
                  const double *bw, double *part, double *dst)
{
    k_gal_dots<<<GAL_NP, BS, 0, s>>>(n, dd, x0, r1, bw, part);
    k_reduce<<<1, 1024, 0, s>>>(part, GAL_MAX * GAL_MAX + GAL_MAX, GAL_NP, dst);
}

void pcg_gal_update(cudaStream_t s, long long n, const GalDirs &dd, const GalCoef &al, const double *x0, double *x)
{
    k_gal_update<<<nblk(n), BS, 0, s>>>(n, dd, al, x0, x);
}

int pcg_nparts() { return NP; }
// blocks of the grid-stride kernels: NP, or as many as have elements
static unsigned nblk(long long n) { return (unsigned)std::min<long long>(NP, (n + BS - 1) / BS); }

static dim3 g3k(const MgDevLevel &L)
{
    return dim3((unsigned)((L.nx + 31) / 32), (unsigned)((L.ny + 7) / 8), (unsigned)((L.nz + KC - 1) / KC));
}
int pcg_stencil_parts(const MgDevLevel &L)
{
    dim3 g = g3k(L);
    return (int)(g.x * g.y * g.z);
}

void pcg_rmax(cudaStream_t s, const MgDevLevel &L0, const double *r, double *part, double *dst)
{
    k_rmax<<<g3k(L0), dim3(32, 8), 0, s>>>(L0, r, part);
    k_max_parts<<<1, 1024, 0, s>>>(part, pcg_stencil_parts(L0), dst);
}

void pcg_gather(cudaStream_t s, const Dims &d, const MgDevLevel &L0, const double *phi_da, const double *pb_da,
                double *x, double *bw)
{
    k_gather<<<dim3((L0.nx + 31) / 32, (L0.ny + 7) / 8, L0.nz), dim3(32, 8), 0, s>>>(d, L0, phi_da, pb_da, x, bw);
}

void pcg_scatter(cudaStream_t s, const Dims &d, const MgDevLevel &L0, const double *x, double *phi_da)
{
    k_scatter<<<dim3((d.NX + 31) / 32, (d.NY + 7) / 8, d.NZ), dim3(32, 8), 0, s>>>(d, L0, x, phi_da);
}

// plane groups per block of the stencil kernels: as many as leave about seven
// 256-thread blocks per SM (k_apply at 256x128x128, 4096 partials: 125 us
// with one group, 111 us with four, the FP64 pipe 88 % active; at 128x64x64, 512 partials, fewer blocks
// than one group gives would leave SMs idle)
static int groups(const MgDevLevel &L0)
{
    const int parts = pcg_stencil_parts(L0);
    return parts >= 4096 ? 4 : parts >= 2048 ? 2 : 1;
}
static dim3 g3g(const MgDevLevel &L0, int g)
{
    dim3 d = g3k(L0);
    d.z = (d.z + g - 1) / g;
    return d;
}

void pcg_resid(cudaStream_t s, const MgDevLevel &L0, const double *bw, const double *x, double *r, double *part,
               double *dst, unsigned *count)
{
    const int np = pcg_stencil_parts(L0), g = groups(L0);
    const dim3 gr = g3g(L0, g), b(32, 8);
    if (g == 4) k_resid<4><<<gr, b, 0, s>>>(L0, bw, x, r, part, np, dst, count);
    else if (g == 2) k_resid<2><<<gr, b, 0, s>>>(L0, bw, x, r, part, np, dst, count);
    else k_resid<1><<<gr, b, 0, s>>>(L0, bw, x, r, part, np, dst, count);
}

void pcg_apply(cudaStream_t s, const MgDevLevel &L0, const double *p, double *q, double *part, PcgScal *sc,
               unsigned *count, int pdl)
{
    const int np = pcg_stencil_parts(L0), g = groups(L0);
    const dim3 gr = g3g(L0, g), b(32, 8);
    if (g == 4) launch_early(pdl, k_apply<4>, gr, b, 0u, s, L0, p, q, part, np, sc, count);
    else if (g == 2) launch_early(pdl, k_apply<2>, gr, b, 0u, s, L0, p, q, part, np, sc, count);
    else launch_early(pdl, k_apply<1>, gr, b, 0u, s, L0, p, q, part, np, sc, count);
}

void pcg_dot(cudaStream_t s, long long n, const double *a, const double *b, double *part, double *dst, unsigned *count)
{
    const unsigned nb = nblk(n);
    k_dot<<<(nb + VB - 1) / VB, BS, 0, s>>>(n, (int)nb, a, b, part, dst, count);
}

void pcg_dot2(cudaStream_t s, long long n, const double *r, const double *z, const double *rold, double *part,
              PcgScal *sc, int restart, unsigned *count, int pdl)
{
    const unsigned nb = nblk(n);
    launch_early(pdl, k_dot2, dim3((nb + VB - 1) / VB), dim3(BS), 0u, s, n, (int)nb, r, z, rold, part, sc, restart, count);
}

void pcg_pupdate(cudaStream_t s, long long n, const double *z, double *p, const PcgScal *sc, int first, int pdl)
{
    const unsigned nb = nblk(n);
    launch_early(pdl, k_pupdate, dim3((nb + VB - 1) / VB), dim3(BS), 0u, s, n, (int)nb, z, p, sc, first);
}

void pcg_xrupdate(cudaStream_t s, long long n, double *x, double *r, double *rold, const double *p,
                  const double *q, PcgScal *sc, double *part, double *host_rr, unsigned *count, int pdl)
{
    const unsigned nb = nblk(n);
    launch_early(pdl, k_xrupdate, dim3((nb + VB - 1) / VB), dim3(BS), 0u, s, n, (int)nb, x, r, rold, p, q, sc, part, host_rr, count);
}

void pcg_reduce(cudaStream_t s, const double *part, int nvals, double *dst, int nper)
{
    k_reduce<<<1, 1024, 0, s>>>(part, nvals, nper > 0 ? nper : NP, dst);
}

void pcg_to_float(cudaStream_t s, long long n, const double *a, float *b) { k_f2<<<nblk(n), BS, 0, s>>>(n, a, b); }
void pcg_to_double(cudaStream_t s, long long n, const float *a, double *b) { k_d2<<<nblk(n), BS, 0, s>>>(n, a, b); }
void pcg_copy(cudaStream_t s, long long n, const double *a, double *b) { k_copy<<<nblk(n), BS, 0, s>>>(n, a, b); }
void pcg_lincomb(cudaStream_t s, long long n, double a, const double *x, double b, const double *y, double *out)
{
    k_lincomb<<<nblk(n), BS, 0, s>>>(n, a, x, b, y, out);
}
