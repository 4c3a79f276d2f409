// k_solve.cu -- implicit viscous / diffusive (Helmholtz) solves and the
// reductions they use.
//
// The operator is the matrix of Velocity_{u,v,w}_form_LHS_matrix /
// Conc_form_LHS_matrix plus the 1/dt diagonal of *_modify_diagonal, applied
// matrix-free: every stencil coefficient is a product of 1-D metric arrays,
// so a row needs the 1-D tables of HelmTab only.  Immersed rows are a gather
// over <= 8 precomputed (column, value) pairs.  The solver is point-Jacobi
// iteration to the reference's test ||b - A x|| <= rtol ||b|| (KSPIBCGS
// without a preconditioner in Solver.c:269-322 reaches the same discrete
// solution); the squared residual norm is reduced in the sweep itself.
#include "turb_internal.cuh"
#include "turb_kernels.cuh"
#include "turb_sum.cuh"

namespace {

constexpr int HBX = 32, HBY = 8, KC = 4;   // 32x8 threads over (i, j), KC planes per thread
constexpr int KCJ = 2;                      // planes per thread of the FP32 Jacobi sweep

// the n partials of one sum, added by the last of `blocks` blocks (of one or
// two launches that share the counter) into *dst
struct SumTo {
    int n;
    unsigned blocks, *count;
    double *dst;
};
__device__ __forceinline__ void sum_to(const double *part, const SumTo &to)
{
    if (last_block(to.count, to.blocks)) sum_parts<1>(part, 0, to.n, to.dst);
}

// FP64 <-> FP32 without the conversion instructions, which run on the FP64
// pipe (two lanes per SM and clock on GB300): normal results are shifted and
// rounded to nearest even on the integer pipe, the others converted
__device__ __forceinline__ float to_f32(double v)
{
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v), e = hi >> 20 & 0x7ffu;
    if (e - 897u > 1150u - 897u) return (float)v;
    unsigned f = (e - 896u) << 23 | (hi & 0xfffffu) << 3 | lo >> 29;
    const unsigned rest = lo & 0x1fffffffu;
    f += rest > 0x10000000u || (rest == 0x10000000u && (f & 1u)) ? 1u : 0u;
    return __uint_as_float(f | (hi & 0x80000000u));
}
__device__ __forceinline__ double to_f64(float v)
{
    const unsigned u = __float_as_uint(v), e = u >> 23 & 0xffu;
    if (e - 1u > 253u) return (double)v;
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
}

__device__ __forceinline__ long long part_index()
{
    return ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
}

// offsets of the six neighbours; an absent neighbour (coefficient 0) is
// redirected to the point itself so that every load stays inside the field
struct Nb {
    long long w, e, s, n, b, f;
};
__device__ __forceinline__ Nb nb_of(const Dims &d, int i, int j, int k)
{
    Nb o;
    o.w = i > 0 ? -1 : 0;
    o.e = i < d.NX - 1 ? 1 : 0;
    o.s = j > 0 ? -(long long)d.PX : 0;
    o.n = j < d.NY - 1 ? (long long)d.PX : 0;
    o.b = k > 0 ? -d.plane : 0;
    o.f = k < d.NZ - 1 ? d.plane : 0;
    return o;
}

__device__ __forceinline__ bool is_stencil(int q, int s)
{
    return (q == 3) ? (s == T_FLUID) : (s == T_FLUID || s == T_BUFFER_SOLID);
}

// (A x)_p and the diagonal of a non-immersed row (rows of *_form_LHS_matrix
// plus 1/dt); coefficients are products of 1-D tables, zero where absent
// axy = apx[i] + apy[j], formed once per (i, j) column by the caller
__device__ __forceinline__ double helm_ax(const Dims &d, const HelmTab &h, int s, double a_dt, double axy,
                                          const double *__restrict__ x, long long p, int i, int j, int k,
                                          double &dg)
{
    if (!is_stencil(h.q, s)) {
        dg = h.ap_solid + a_dt;
        return dg * x[p];
    }
    Nb o = nb_of(d, i, j, k);
    dg = axy + (h.apz[k] + a_dt);
    double acc = dg * x[p];
    acc = fma(h.aw[i], x[p + o.w], acc);
    acc = fma(h.ae[i], x[p + o.e], acc);
    acc = fma(h.as[j], x[p + o.s], acc);
    acc = fma(h.an[j], x[p + o.n], acc);
    acc = fma(h.ab[k], x[p + o.b], acc);
    acc = fma(h.af[k], x[p + o.f], acc);
    return acc;
}

__global__ void k_helm_apply(Dims d, HelmTab h, const uint8_t *__restrict__ st, double a_dt,
                             const double *__restrict__ x, double *__restrict__ y)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= d.NX || j >= d.NY) return;
    const double axy = h.apx[i] + h.apy[j];
    for (int kk = 0; kk < KC; kk++) {
        int k = blockIdx.z * KC + kk;
        if (k >= d.NZ) break;
        long long p = d.at(i, j, k);
        int s = st[p];
        if (s == T_IMMERSED) continue;
        double dg;
        y[p] = helm_ax(d, h, s, a_dt, axy, x, p, i, j, k, dg);
    }
}

// immersed rows: y = diag*x_im + sum val*x_col
__global__ void k_ib_apply(IbDev ib, const double *__restrict__ x, double *__restrict__ y)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ib.n) return;
    long long im = ib.im[t];
    double acc = ib.diag[t] * x[im];
    int c = ib.cnt[t];
    for (int g = 0; g < c; g++) acc += ib.val[t * 8 + g] * x[ib.col[t * 8 + g]];
    y[im] = acc;
}

// one Jacobi sweep xn = x + (b - A x)/diag, partial sums of |b - A x|^2.  On
// small grids (AHEAD) latency bounds it: the KC planes' loads are in flight
// together and their chains of FP64 operations, a division each, interleave
// (two FP64 steps at 64x32x32: 13.32 -> 13.07 ms)
template <bool AHEAD>
__global__ void __launch_bounds__(HBX *HBY) k_helm_jacobi(Dims d, HelmTab h, const uint8_t *__restrict__ st, double a_dt,
                              const double *__restrict__ b, const double *__restrict__ x,
                              double *__restrict__ xn, double *__restrict__ part, const SumTo to)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    double r2 = 0.0;
    if (i < d.NX && j < d.NY) {
        const double axy = h.apx[i] + h.apy[j];
        if (AHEAD) {
            const int k0 = blockIdx.z * KC;
            double ax[KC], dg[KC], xc[KC], bc[KC];
            int sv[KC];
#pragma unroll
            for (int kk = 0; kk < KC; kk++) {   // planes past the last are the last one again, not stored
                const int k = min(k0 + kk, d.NZ - 1);
                const long long p = d.at(i, j, k);
                sv[kk] = st[p];
                xc[kk] = x[p];
                bc[kk] = b[p];
                ax[kk] = helm_ax(d, h, sv[kk], a_dt, axy, x, p, i, j, k, dg[kk]);
            }
#pragma unroll
            for (int kk = 0; kk < KC; kk++) {
                const double r = bc[kk] - ax[kk], v = xc[kk] + r / dg[kk];
                if (k0 + kk < d.NZ && sv[kk] != T_IMMERSED) {
                    xn[d.at(i, j, k0 + kk)] = v;
                    r2 = fma(r, r, r2);
                }
            }
        } else {
            for (int kk = 0; kk < KC; kk++) {
                int k = blockIdx.z * KC + kk;
                if (k >= d.NZ) break;
                long long p = d.at(i, j, k);
                int s = st[p];
                if (s == T_IMMERSED) continue;
                double dg, ax = helm_ax(d, h, s, a_dt, axy, x, p, i, j, k, dg);
                double r = b[p] - ax;
                xn[p] = x[p] + r / dg;
                r2 = fma(r, r, r2);
            }
        }
    }
    double bs[1];
    block_sum256<1>({r2}, bs);
    if (threadIdx.x == 0 && threadIdx.y == 0) part[part_index()] = bs[0];
    sum_to(part, to);
}

__global__ void k_ib_jacobi(IbDev ib, const double *__restrict__ b, const double *__restrict__ x,
                            double *__restrict__ xn, double *__restrict__ part, long long part0, const SumTo to)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    double r2 = 0.0;
    if (t < ib.n) {
        long long im = ib.im[t];
        double acc = ib.diag[t] * x[im];
        int c = ib.cnt[t];
        for (int g = 0; g < c; g++) acc += ib.val[t * 8 + g] * x[ib.col[t * 8 + g]];
        double r = b[im] - acc;
        xn[im] = x[im] + r / ib.diag[t];
        r2 = r * r;
    }
    double bs[1];
    block_sum256<1>({r2}, bs);
    if (threadIdx.x == 0) part[part0 + blockIdx.x] = bs[0];
    sum_to(part, to);
}

// ---- mixed-precision defect correction -----------------------------------
// x += e over the whole field (FP64 accumulation of the FP32 correction of a
// single sweep)
__global__ void k_add_corr(long long n, double *__restrict__ x, const float *__restrict__ e)
{
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        x[p] = x[p] + (double)e[p];
}

// r = b - A x in FP64, rounded to FP32 for the inner solve; |r|^2; and the
// inner solve's first sweep, e = r / diag (from e = 0), whose FP32 work is free
// here.  The FP64 pipe bounds this kernel on large grids, so the row is
// accumulated as -(diag x - b + sum a_nb x_nb) (no separate subtraction),
// apz[k] + 1/dt is formed once per plane of the block and r is rounded on the
// integer pipe: nine FP64 operations per point.  On small grids (G = 0)
// latency does: the KC planes' loads are all in flight before the first row is
// formed (98 registers; on large grids fewer warps then cost more than the
// latency: 975 us against 715 at 513x257x257).  The last block adds the
// partial sums.  adt: 1/dt for the sweeps, whose captured graphs outlive a
// time step of one length.
struct ResidRow {
    double axy, aw, ae, as, an;
    float afx, afy;
};
__device__ __forceinline__ void resid_store(const HelmTab &h, const HelmTabF &hf, const ResidRow &w, double a_dt, double zdt, int s,
                                            int k, double xc, double bc, double xw, double xe, double xs, double xn, double xb,
                                            double xf, float *rf, float *e0, double &r2)
{
    const bool stn = is_stencil(h.q, s);
    double r;
    if (!stn) {
        r = bc - (h.ap_solid + a_dt) * xc;
    } else {
        double acc = fma(w.axy + zdt, xc, -bc);
        acc = fma(w.aw, xw, acc);
        acc = fma(w.ae, xe, acc);
        acc = fma(w.as, xs, acc);
        acc = fma(w.an, xn, acc);
        acc = fma(h.ab[k], xb, acc);
        acc = fma(h.af[k], xf, acc);
        r = -acc;
    }
    const float rv = to_f32(r), a_dtf = (float)a_dt;
    const float dg = stn ? __fadd_rn(__fadd_rn(__fadd_rn(w.afx, w.afy), hf.apz[k]), a_dtf) : __fadd_rn(hf.ap_solid, a_dtf);
    *rf = rv;
    *e0 = __fmul_rn(rv, __frcp_rn(dg));
    r2 = fma(r, r, r2);
}

// G: groups of KC planes a block marches, G partial sums (those of G blocks of
// one group); 0: one group with AHEAD loads
template <int G>
__global__ void __launch_bounds__(HBX *HBY, G ? 4 : 2) k_helm_resid64(Dims d, HelmTab h, HelmTabF hf, const uint8_t *__restrict__ st, double a_dt,
                               const double *__restrict__ b, const double *__restrict__ x,
                               float *__restrict__ rf, float *__restrict__ e0, float *__restrict__ adt, double *__restrict__ part,
                               const SumTo to)
{
    constexpr int NG = G ? G : 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k0 = blockIdx.z * KC * NG;
    __shared__ double zdt[KC * NG];
    {
        int t = threadIdx.y * blockDim.x + threadIdx.x, k = k0 + t;
        if (t < KC * NG) zdt[t] = k < d.NZ ? h.apz[k] + a_dt : 0.0;
        if (t == 0 && part_index() == 0) *adt = (float)a_dt;   // for the sweeps
    }
    __syncthreads();
    double r2[NG] = {};
    pdl_trigger();   // the immersed rows' kernel (disjoint points) may start at once
    if (i < d.NX && j < d.NY) {
        const long long pj = d.at(i, j, 0);
        const int ow = i > 0 ? -1 : 0, oe = i < d.NX - 1 ? 1 : 0;
        const int os = j > 0 ? -(int)d.PX : 0, on = j < d.NY - 1 ? (int)d.PX : 0;
        const ResidRow w{h.apx[i] + h.apy[j], h.aw[i], h.ae[i], h.as[j], h.an[j], hf.apx[i], hf.apy[j]};
        if (G == 0) {
            // planes past the last are the last one again, not stored; so is the
            // neighbour beyond an end plane (its coefficient is zero)
            double xc[KC + 2], xw[KC], xe[KC], xs[KC], xn[KC], bc[KC];
            int sv[KC];
            xc[0] = x[pj + max(k0 - 1, 0) * d.plane];
#pragma unroll
            for (int kk = 0; kk < KC; kk++) {
                const long long p = pj + min(k0 + kk, d.NZ - 1) * d.plane;
                sv[kk] = st[p];
                xc[kk + 1] = x[p];
                xw[kk] = x[p + ow];
                xe[kk] = x[p + oe];
                xs[kk] = x[p + os];
                xn[kk] = x[p + on];
                bc[kk] = b[p];
            }
            xc[KC + 1] = x[pj + min(k0 + KC, d.NZ - 1) * d.plane];
#pragma unroll
            for (int kk = 0; kk < KC; kk++) {
                const int k = k0 + kk;
                const long long p = pj + k * d.plane;
                if (k < d.NZ && sv[kk] != T_IMMERSED)
                    resid_store(h, hf, w, a_dt, zdt[kk], sv[kk], k, xc[kk + 1], bc[kk], xw[kk], xe[kk], xs[kk], xn[kk], xc[kk],
                                xc[kk + 2], rf + p, e0 + p, r2[0]);
            }
        } else {
            long long p = pj + k0 * d.plane;
            double xc = x[p], xb = k0 > 0 ? x[p - d.plane] : xc;
#pragma unroll
            for (int g = 0; g < NG; g++) {
                for (int kk = 0; kk < KC; kk++, p += d.plane) {
                    const int k = k0 + g * KC + kk;
                    if (k >= d.NZ) break;
                    const double xf = k < d.NZ - 1 ? x[p + d.plane] : xc;
                    const int s = st[p];
                    if (s != T_IMMERSED)
                        resid_store(h, hf, w, a_dt, zdt[g * KC + kk], s, k, xc, b[p], x[p + ow], x[p + oe], x[p + os], x[p + on],
                                    xb, xf, rf + p, e0 + p, r2[g]);
                    xb = xc;
                    xc = xf;
                }
            }
        }
    }
    double bs[NG];
    block_sum256<NG>(r2, bs);
    if (threadIdx.x == 0 && threadIdx.y == 0)
#pragma unroll
        for (int g = 0; g < NG; g++) {
            const int bz = blockIdx.z * NG + g;
            if (bz * KC < d.NZ) part[((long long)bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = bs[g];
        }
    sum_to(part, to);
}

__global__ void k_ib_resid64(IbDev ib, IbDevF ibf, const double *__restrict__ b, const double *__restrict__ x,
                             float *__restrict__ rf, float *__restrict__ e0, double *__restrict__ part, long long part0,
                             const SumTo to)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    double r2 = 0.0;
    if (t < ib.n) {
        long long im = ib.im[t];
        double acc = ib.diag[t] * x[im];
        int c = ib.cnt[t];
        for (int g = 0; g < c; g++) acc += ib.val[t * 8 + g] * x[ib.col[t * 8 + g]];
        double r = b[im] - acc;
        rf[im] = (float)r;
        e0[im] = (float)r * __frcp_rn(ibf.diag[t]);
        r2 = r * r;
    }
    double bs[1];
    block_sum256<1>({r2}, bs);
    if (threadIdx.x == 0) part[part0 + blockIdx.x] = bs[0];
    sum_to(part, to);
    pdl_wait();   // as in k_ib_jac32: end after the stencil residual
}

// inner FP32 Jacobi sweep on A e = r (after the first, which the residual
// does), four points of a row per thread: e, r, status and the j+-1 / k+-1
// neighbours are 16-byte (4-byte for status) loads, the x tables are padded to
// the pitch.  The last sweep (LAST) adds its result to x instead of storing
// it: 25 bytes per point where the sweep and the addition moved 33.  Immersed
// points are left to k_ib_jac32 (not written here, so the two kernels may
// overlap); pad columns (i >= NX) are not written.  e and
// x, which kernels just before write, are not __restrict__: nothing reads them
// before pdl_wait.
// four blocks of 32 x 8 per SM (64 registers): measured 17 % faster at
// 513x257x257 than the three that 76 registers allow
template <bool LAST>
__global__ void __launch_bounds__(HBX *HBY, 4) k_helm_jac32v(Dims d, HelmTabF h, const uint8_t *__restrict__ st, const float *adt,
                              const float *__restrict__ r, const float *e, float *en, double *x)
{
    const int i0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x), j = blockIdx.y * blockDim.y + threadIdx.y;
    pdl_wait();
    pdl_trigger();   // the immersed rows' kernel, which reads e too, may start
    if (i0 >= d.NX || j >= d.NY) return;
    const float a_dt = *adt;
    const float4 apx = *reinterpret_cast<const float4 *>(h.apx + i0);
    const float4 aw = *reinterpret_cast<const float4 *>(h.aw + i0);
    const float4 ae = *reinterpret_cast<const float4 *>(h.ae + i0);
    const float apxv[4] = {apx.x, apx.y, apx.z, apx.w}, awv[4] = {aw.x, aw.y, aw.z, aw.w};
    const float aev[4] = {ae.x, ae.y, ae.z, ae.w};
    const float apyj = h.apy[j], asj = h.as[j], anj = h.an[j];
    const int nvalid = min(4, d.NX - i0);
    for (int kk = 0; kk < KCJ; kk++) {
        const int k = blockIdx.z * KCJ + kk;
        if (k >= d.NZ) break;
        const long long p = d.at(i0, j, k);
        const uchar4 s4 = *reinterpret_cast<const uchar4 *>(st + p);
        const int sv[4] = {s4.x, s4.y, s4.z, s4.w};
        const float4 r4 = *reinterpret_cast<const float4 *>(r + p);
        const float rv[4] = {r4.x, r4.y, r4.z, r4.w};
        const float apzk = h.apz[k], abk = h.ab[k], afk = h.af[k];
        float out[4];
        const float4 e4 = *reinterpret_cast<const float4 *>(e + p);
        const float ev[4] = {e4.x, e4.y, e4.z, e4.w};
        const float xw = i0 > 0 ? e[p - 1] : ev[0];
        const float xe = i0 + 4 < d.NX ? e[p + 4] : ev[3];
        const float4 s_ = j > 0 ? *reinterpret_cast<const float4 *>(e + p - d.PX) : e4;
        const float4 n_ = j < d.NY - 1 ? *reinterpret_cast<const float4 *>(e + p + d.PX) : e4;
        const float4 b_ = k > 0 ? *reinterpret_cast<const float4 *>(e + p - d.plane) : e4;
        const float4 f_ = k < d.NZ - 1 ? *reinterpret_cast<const float4 *>(e + p + d.plane) : e4;
        const float sv_[4] = {s_.x, s_.y, s_.z, s_.w}, nv_[4] = {n_.x, n_.y, n_.z, n_.w};
        const float bv_[4] = {b_.x, b_.y, b_.z, b_.w}, fv_[4] = {f_.x, f_.y, f_.z, f_.w};
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const bool stn = is_stencil(h.q, sv[t]);
            const float dg = stn ? __fadd_rn(__fadd_rn(__fadd_rn(apxv[t], apyj), apzk), a_dt)
                                 : __fadd_rn(h.ap_solid, a_dt);
            float acc = __fmul_rn(dg, ev[t]);
            if (stn) {
                acc = __fmaf_rn(awv[t], t == 0 ? xw : ev[t - 1], acc);
                acc = __fmaf_rn(aev[t], t == 3 ? xe : ev[t + 1], acc);
                acc = __fmaf_rn(asj, sv_[t], acc);
                acc = __fmaf_rn(anj, nv_[t], acc);
                acc = __fmaf_rn(abk, bv_[t], acc);
                acc = __fmaf_rn(afk, fv_[t], acc);
            }
            out[t] = __fmaf_rn(__fadd_rn(rv[t], -acc), __frcp_rn(dg), ev[t]);
        }
        const bool ib4 = sv[0] == T_IMMERSED || sv[1] == T_IMMERSED || sv[2] == T_IMMERSED || sv[3] == T_IMMERSED;
        const bool all = nvalid == 4 && !ib4;
        if (LAST) {
            if (all) {
                double2 *xp = reinterpret_cast<double2 *>(x + p);
                double2 lo = xp[0], hi = xp[1];
                lo.x += to_f64(out[0]);
                lo.y += to_f64(out[1]);
                hi.x += to_f64(out[2]);
                hi.y += to_f64(out[3]);
                xp[0] = lo;
                xp[1] = hi;
            } else {
                for (int t = 0; t < nvalid; t++)
                    if (sv[t] != T_IMMERSED) x[p + t] += (double)out[t];
            }
        } else if (all) {
            *reinterpret_cast<float4 *>(en + p) = make_float4(out[0], out[1], out[2], out[3]);
        } else {
            for (int t = 0; t < nvalid; t++)
                if (sv[t] != T_IMMERSED) en[p + t] = out[t];
        }
    }
}

// The same sweep (not the first one) marching along k: a block of 32 x 8
// threads owns a tile of 128 x 8 points of every plane of a chunk of JZ
// planes.  Each thread keeps its four points of planes k-1, k, k+1 in
// registers (e of plane k+1 is loaded while plane k is computed); the x and
// y neighbours come from the plane-k tile in shared memory, whose halo rows
// j-1, j+8 and columns are loaded by the edge threads.  e is read from
// memory about once per sweep instead of once per neighbour, and every
// point's arithmetic and neighbour substitutions are k_helm_jac32v's, so the
// results are the same bits.
constexpr int JZ = 16;                 // planes per block
constexpr int JTX = 4 * HBX + 2;       // tile row: 128 points and two halo columns
__global__ void __launch_bounds__(HBX *HBY, 3) k_helm_jac32z(Dims d, HelmTabF h, const uint8_t *__restrict__ st,
                                                          const float *__restrict__ adt, const float *__restrict__ r,
                                                          const float *__restrict__ e, float *__restrict__ en)
{
    __shared__ float tile[HBY + 2][JTX];
    const float a_dt = *adt;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int i0 = 4 * (blockIdx.x * HBX + tx), j = blockIdx.y * HBY + ty;
    const int k0 = blockIdx.z * JZ, k1 = min(k0 + JZ, d.NZ);
    const bool act = i0 < d.NX && j < d.NY;
    const int nvalid = act ? min(4, d.NX - i0) : 0;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float apxv[4] = {}, awv[4] = {}, aev[4] = {};
    float apyj = 0.f, asj = 0.f, anj = 0.f;
    if (act) {
        const float4 apx = *reinterpret_cast<const float4 *>(h.apx + i0);
        const float4 aw = *reinterpret_cast<const float4 *>(h.aw + i0);
        const float4 ae = *reinterpret_cast<const float4 *>(h.ae + i0);
        apxv[0] = apx.x; apxv[1] = apx.y; apxv[2] = apx.z; apxv[3] = apx.w;
        awv[0] = aw.x; awv[1] = aw.y; awv[2] = aw.z; awv[3] = aw.w;
        aev[0] = ae.x; aev[1] = ae.y; aev[2] = ae.z; aev[3] = ae.w;
        apyj = h.apy[j]; asj = h.as[j]; anj = h.an[j];
    }
    const long long pj = act ? d.at(i0, j, 0) : 0;
    // the edge threads also load a halo row (j-1 for the first row of the
    // block, j+1 for the last) and a halo column (left / right of the tile)
    const int jh = ty == 0 ? j - 1 : (ty == HBY - 1 ? j + 1 : -1);
    const bool hrow = act && jh >= 0 && jh < d.NY;
    const long long ph = hrow ? d.at(i0, jh, 0) : 0;
    const bool hl = act && tx == 0 && i0 > 0, hr_ = act && tx == HBX - 1 && i0 + 4 < d.NX;
    auto in_k = [&](int k) { return act && k >= 0 && k < d.NZ; };
    auto ld4 = [&](const float *a, long long base, int k) -> float4 {
        return in_k(k) ? *reinterpret_cast<const float4 *>(a + base + (long long)k * d.plane) : z4;
    };
    // plane k0 and the planes around it; the rest is loaded one plane ahead
    float4 eb = ld4(e, pj, k0 - 1), ec = ld4(e, pj, k0), ef = ld4(e, pj, k0 + 1);
    float4 rc = ld4(r, pj, k0);
    uchar4 sc = in_k(k0) ? *reinterpret_cast<const uchar4 *>(st + pj + (long long)k0 * d.plane) : make_uchar4(0, 0, 0, 0);
    float4 hc = (hrow && k0 < d.NZ) ? ld4(e, ph, k0) : z4;
    float xlc = hl ? e[pj + (long long)k0 * d.plane - 1] : 0.f, xrc = hr_ ? e[pj + (long long)k0 * d.plane + 4] : 0.f;
    for (int k = k0; k < k1; k++) {
        const float ev[4] = {ec.x, ec.y, ec.z, ec.w};
        float *row = &tile[ty + 1][1 + 4 * tx];
        row[0] = ev[0]; row[1] = ev[1]; row[2] = ev[2]; row[3] = ev[3];
        if (hrow) {
            float *hrw = &tile[ty == 0 ? 0 : HBY + 1][1 + 4 * tx];
            hrw[0] = hc.x; hrw[1] = hc.y; hrw[2] = hc.z; hrw[3] = hc.w;
        }
        if (hl) tile[ty + 1][0] = xlc;
        if (hr_) tile[ty + 1][JTX - 1] = xrc;
        __syncthreads();
        // the next plane's loads, in flight while this plane is computed
        const int kn = k + 1;
        const float4 ef2 = ld4(e, pj, kn + 1), rn = ld4(r, pj, kn);
        const uchar4 sn = in_k(kn) ? *reinterpret_cast<const uchar4 *>(st + pj + (long long)kn * d.plane)
                                   : make_uchar4(0, 0, 0, 0);
        const float4 hn = (hrow && kn < d.NZ) ? ld4(e, ph, kn) : z4;
        const float xln = (hl && kn < d.NZ) ? e[pj + (long long)kn * d.plane - 1] : 0.f;
        const float xrn = (hr_ && kn < d.NZ) ? e[pj + (long long)kn * d.plane + 4] : 0.f;
        if (act) {
            const long long p = pj + (long long)k * d.plane;
            const int sv[4] = {sc.x, sc.y, sc.z, sc.w};
            const float rv[4] = {rc.x, rc.y, rc.z, rc.w};
            const float apzk = h.apz[k], abk = h.ab[k], afk = h.af[k];
            const float xw = i0 > 0 ? tile[ty + 1][4 * tx] : ev[0];
            const float xe = i0 + 4 < d.NX ? tile[ty + 1][4 * tx + 5] : ev[3];
            float sv_[4], nv_[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                sv_[t] = j > 0 ? tile[ty][1 + 4 * tx + t] : ev[t];
                nv_[t] = j < d.NY - 1 ? tile[ty + 2][1 + 4 * tx + t] : ev[t];
            }
            const float4 b_ = k > 0 ? eb : ec, f_ = k < d.NZ - 1 ? ef : ec;
            const float bv_[4] = {b_.x, b_.y, b_.z, b_.w}, fv_[4] = {f_.x, f_.y, f_.z, f_.w};
            float out[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const bool stn = is_stencil(h.q, sv[t]);
                const float dg = stn ? __fadd_rn(__fadd_rn(__fadd_rn(apxv[t], apyj), apzk), a_dt)
                                     : __fadd_rn(h.ap_solid, a_dt);
                float acc = __fmul_rn(dg, ev[t]);
                if (stn) {
                    acc = __fmaf_rn(awv[t], t == 0 ? xw : ev[t - 1], acc);
                    acc = __fmaf_rn(aev[t], t == 3 ? xe : ev[t + 1], acc);
                    acc = __fmaf_rn(asj, sv_[t], acc);
                    acc = __fmaf_rn(anj, nv_[t], acc);
                    acc = __fmaf_rn(abk, bv_[t], acc);
                    acc = __fmaf_rn(afk, fv_[t], acc);
                }
                out[t] = __fmaf_rn(__fadd_rn(rv[t], -acc), __frcp_rn(dg), ev[t]);
            }
            if (nvalid == 4) {
                *reinterpret_cast<float4 *>(en + p) = make_float4(out[0], out[1], out[2], out[3]);
            } else {
                for (int t = 0; t < nvalid; t++) en[p + t] = out[t];
            }
        }
        __syncthreads();
        eb = ec;
        ec = ef;
        ef = ef2;
        rc = rn;
        sc = sn;
        hc = hn;
        xlc = xln;
        xrc = xrn;
    }
}

__global__ void k_ib_jac32(IbDevF ib, const float *__restrict__ r, const float *__restrict__ e,
                           float *__restrict__ en, double *__restrict__ x)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ib.n) {
        long long im = ib.im[t];
        float inv = __frcp_rn(ib.diag[t]);
        float acc = ib.diag[t] * e[im];
        int c = ib.cnt[t];
        for (int g = 0; g < c; g++) acc += ib.val[t * 8 + g] * e[ib.col[t * 8 + g]];
        const float v = fmaf(r[im] - acc, inv, e[im]);
        if (x) x[im] += (double)v;
        else en[im] = v;
    }
    // launched as a programmatic dependent of the stencil sweep (which
    // writes the other points): end only after it has completed, so
    // that the kernels after this one see both
    pdl_wait();
}

inline dim3 hgrid(const Dims &d)
{
    return dim3((unsigned)((d.NX + HBX - 1) / HBX), (unsigned)((d.NY + HBY - 1) / HBY),
                (unsigned)((d.NZ + KC - 1) / KC));
}

constexpr int NPART = 1024;

__global__ void k_norm2(long long n, long long stride, const double *__restrict__ x, double *__restrict__ part, const SumTo to)
{
    double v = 0.0;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride)
        v += x[p] * x[p];
    double s[1];
    block_sum256<1>({v}, s);
    if (threadIdx.x == 0) part[blockIdx.x] = s[0];
    sum_to(part, to);
}

}  // namespace

long long helm_parts(const Dims &d)
{
    dim3 g = hgrid(d);
    return (long long)g.x * g.y * g.z;
}

void launch_helm_apply(cudaStream_t s, const Dims &d, const HelmTab &h, const uint8_t *st, double a_dt,
                       const double *x, double *y, const IbDev &ib)
{
    k_helm_apply<<<hgrid(d), dim3(HBX, HBY), 0, s>>>(d, h, st, a_dt, x, y);
    if (ib.n > 0) k_ib_apply<<<(ib.n + 255) / 256, 256, 0, s>>>(ib, x, y);
}

// part must hold helm_parts(d) + (ib.n+255)/256 entries; |r|^2 goes to *dst
void launch_helm_jacobi(cudaStream_t s, const Dims &d, const HelmTab &h, const uint8_t *st, double a_dt,
                        const double *b, const double *x, double *xn, const IbDev &ib, double *part,
                        unsigned *count, double *dst, int nsm)
{
    const long long hp = helm_parts(d);
    const unsigned nib = (unsigned)((ib.n + 255) / 256);
    const SumTo to{(int)(hp + nib), (unsigned)hp + nib, count, dst};
    const auto k = hp <= 2 * nsm ? k_helm_jacobi<true> : k_helm_jacobi<false>;
    k<<<hgrid(d), dim3(HBX, HBY), 0, s>>>(d, h, st, a_dt, b, x, xn, part, to);
    if (ib.n > 0) k_ib_jacobi<<<nib, 256, 0, s>>>(ib, b, x, xn, part, hp, to);
}

// |x|^2 to *dst
void launch_norm2(cudaStream_t s, long long n, const double *x, double *part, unsigned *count, double *dst)
{
    // blocks without elements would add zeros
    const long long want = (n + 255) / 256;
    const int nb = (int)(want < NPART ? (want > 0 ? want : 1) : NPART);
    k_norm2<<<nb, 256, 0, s>>>(n, (long long)NPART * 256, x, part, SumTo{nb, (unsigned)nb, count, dst});
}

void launch_add_corr(cudaStream_t s, long long n, double *x, const float *e)
{
    k_add_corr<<<1216, 256, 0, s>>>(n, x, e);
}

// |r|^2 goes to *dst, the first sweep's result to e0, 1/dt for the others to *adt
void launch_helm_resid64(cudaStream_t s, const Dims &d, const HelmTab &h, const HelmTabF &hf, const uint8_t *st, double a_dt,
                         const double *b, const double *x, float *rf, float *e0, float *adt, const IbDev &ib,
                         const IbDevF &ibf, double *part, unsigned *count, double *dst, int nsm, int pdl)
{
    const long long hp = helm_parts(d);
    const unsigned nib = (unsigned)((ib.n + 255) / 256);
    // groups per block: as many as leave about seven blocks per SM
    const int g = hp >= 4096 ? 4 : hp >= 2048 ? 2 : hp > 2 * nsm ? 1 : 0;
    dim3 gr = hgrid(d);
    if (g) gr.z = (gr.z + g - 1) / g;
    const SumTo to{(int)(hp + nib), gr.x * gr.y * gr.z + nib, count, dst};
    const auto k = g == 4 ? k_helm_resid64<4> : g == 2 ? k_helm_resid64<2> : g == 1 ? k_helm_resid64<1> : k_helm_resid64<0>;
    k<<<gr, dim3(HBX, HBY), 0, s>>>(d, h, hf, st, a_dt, b, x, rf, e0, adt, part, to);
    // the immersed rows beside it: they read nothing that it writes, write
    // only immersed points and end with pdl_wait
    if (ib.n > 0) launch_early(pdl, k_ib_resid64, dim3(nib), dim3(256), 0u, s, ib, ibf, b, x, rf, e0, part, hp, to);
}

// The sweep after the first ones: from e to en, or (x given) added to x.
// alone: the kernel ahead of it on the stream is not a sweep.  marching 1: the
// sweeps but the last march along k through shared-memory plane tiles
// (k_helm_jac32z); 0: k_helm_jac32v throughout
void launch_helm_jac32(cudaStream_t s, const Dims &d, const HelmTabF &h, const uint8_t *st, const float *adt,
                       const float *r, const float *e, float *en, double *x, const IbDevF &ib, int alone, int marching,
                       int pdl)
{
    dim3 g((unsigned)((d.NX + 4 * HBX - 1) / (4 * HBX)), (unsigned)((d.NY + HBY - 1) / HBY),
           (unsigned)((d.NZ + KCJ - 1) / KCJ));
    if (!x && marching) {
        dim3 gz((unsigned)((d.NX + 4 * HBX - 1) / (4 * HBX)), (unsigned)((d.NY + HBY - 1) / HBY),
                (unsigned)((d.NZ + JZ - 1) / JZ));
        k_helm_jac32z<<<gz, dim3(HBX, HBY), 0, s>>>(d, h, st, adt, r, e, en);
        // k_helm_jac32z writes placeholders at immersed points: the immersed
        // rows go after it in plain stream order
        if (ib.n > 0) k_ib_jac32<<<(ib.n + 255) / 256, 256, 0, s>>>(ib, r, e, en, x);
        return;
    }
    const auto k = x ? k_helm_jac32v<true> : k_helm_jac32v<false>;
    if (alone || marching) k<<<g, dim3(HBX, HBY), 0, s>>>(d, h, st, adt, r, e, en, x);
    else launch_early(pdl, k, g, dim3(HBX, HBY), 0u, s, d, h, st, adt, r, e, en, x);
    if (ib.n > 0) launch_early(pdl, k_ib_jac32, dim3((ib.n + 255) / 256), dim3(256), 0u, s, ib, r, e, en, x);
}
