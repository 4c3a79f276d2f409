// k_eno.cu -- ENO convection: the line driver restated around
// ENO_compute_convective_terms (ENO.c:103-245) and the ghost-cell rules of
// Velocity_{u,v,w}_ENO_ghost_cells / Conc_ENO_ghost_cells.
//
// Work per (quantity, direction) pass, conv = Vx dq/dx (+ Vy dq/dy) (+ Vz dq/dz):
//  * x: one block per x-line; the line buffer (interior + ghosts) is staged in
//       shared memory and each divided difference is formed once;
//  * y, z: one thread per segment of a line walking along it with a sliding
//       register window (loads coalesced across i); each step forms one new
//       D1, D2, D3.
// Every divided difference rounds as the IEEE division on the same operands as
// the reference, and every sum and product as if rounded one by one, so the
// stencil choices and fluxes are bit-identical to the reference's C.
//
// The FP64 pipe (488 G operations/s) bounds every pass: 0.16 ms of it per 10
// operations at 256x128x128 against 20 us of memory traffic.  So what need not
// be an FP64 operation is not one: magnitude and sign tests, zero and range
// tests are integer operations on the words (dwords, turb_div.cuh); weights of
// 1/2 become one sum and an exact scaling; on a uniform power-of-two spacing
// quotients are scalings and the products with g2, g3 ride in an FMA.
// Measured FP64-pipe instructions per point at 512x256x256: y passes 11 (the
// velocity a field) and 18 (a transpose), z 11 and 15, x 10 and 14 (15 and 21 to
// 22 before, at 256x128x128).  Us per pass, x and y/z, before and after:
// 128x64x64 32 / 128 -> 23 / 29, 256x128x128 196 / 217 -> 121 / 142, 512x256x256
// 1400 / 1500 -> 901 / 991, the FP64 pipe 75-84 % active at 256x128x128 and
// 80-85 % at 512x256x256.
#include <algorithm>
#include <type_traits>

#include "turb_internal.cuh"
#include "turb_kernels.cuh"
#include "turb_div.cuh"

namespace {

__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dadd_rn(a, -b); }
__device__ __forceinline__ double ml(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dv(double a, double b) { return __ddiv_rn(a, b); }

// a / h rounded to nearest: IEEE division or the form of the spacing (EnoDiv)
__device__ __forceinline__ double dd(const EnoTab &T, double a, const EnoDiv &t)
{
    if (!T.fastdiv) return dv(a, t.h);
    if (t.form == 2) return div_by_spacing_2t(a, t.h, t.y, t.yl);
    if (t.form == 1) return ml(a, t.y);
    return div_by_spacing(a, t.h, t.y, t.yl);
}

__device__ __forceinline__ double interp4(double q0, double q1, double q2, double q3, double wx0,
                                          double wx1, double wy0, double wy1)
{
    double qt = ad(ml(wx0, q2), ml(wx1, q3));
    double qb = ad(ml(wx0, q0), ml(wx1, q1));
    return ad(ml(wy0, qb), ml(wy1, qt));
}

// |a| <= |b| on the integer pipe (a DSETP costs as much as a DADD): for
// numbers and infinities the bit patterns without the sign order as the
// magnitudes; false when either is NaN, as the comparison (a NaN a lies above
// every b that is not; a NaN b is ruled out by its high word, arithmetic
// makes no NaN with 0x7ff00000 there)
__device__ __forceinline__ bool abs_le(double a, double b)
{
    const DWords x = dwords(a), y = dwords(b);
    const unsigned xh = x.hi & 0x7fffffffu, yh = y.hi & 0x7fffffffu;
    return (xh < yh || (xh == yh && x.lo <= y.lo)) && yh <= 0x7ff00000u;
}
// v > 0 for a number (a NaN counts as positive: its flux is NaN either way)
__device__ __forceinline__ bool positive(double v)
{
    const DWords w = dwords(v);
    return (int)w.hi > 0 || (w.hi == 0u && w.lo != 0u);
}

// zero, or a binary exponent in [-959, 960]: sums, halves and quarters of
// such values are exact scalings of each other
__device__ __forceinline__ bool scalable(double a)
{
    const DWords w = dwords(a);
    return (w.hi & 0x7ff00000u) - 0x04000000u < 0x78000000u || dw_zero(w);
}

// kept out of line: predicated off, its instructions would still pass through
// the FP64 pipe
__device__ __noinline__ double interp4_call(double q0, double q1, double q2, double q3, double wx0, double wx1,
                                            double wy0, double wy1)
{
    return interp4(q0, q1, q2, q3, wx0, wx1, wy0, wy1);
}

// interp4 with inner weights 1/2: RN(RN(q0/2) + RN(q1/2)) = RN(q0 + q1)/2, so
// the halves move into the outer weights (wy.h*: BIL 2, five FP64 operations
// instead of nine) or, those 1/2 too, into one exact quarter (BIL 1, four)
enum { ADV_FIELD = 0, ADV_HALF = 1, ADV_HALF_X = 2, ADV_BILINEAR = 3 };
template <int BIL>
__device__ __forceinline__ double interp(double q0, double q1, double q2, double q3, const AdvSrc &a, int ix, int iy)
{
    if (BIL != ADV_BILINEAR && scalable(q0) && scalable(q1) && scalable(q2) && scalable(q3)) {
        const double s0 = ad(q0, q1), s1 = ad(q2, q3);
        return BIL == ADV_HALF ? ml(0.25, ad(s0, s1)) : ad(ml(a.wy.h0[iy], s0), ml(a.wy.h1[iy], s1));
    }
    if (BIL == ADV_BILINEAR)
        return interp4(q0, q1, q2, q3, a.wx.w0[ix], a.wx.w1[ix], a.wy.w0[iy], a.wy.w1[iy]);
    return interp4_call(q0, q1, q2, q3, a.wx.w0[ix], a.wx.w1[ix], a.wy.w0[iy], a.wy.w1[iy]);
}

// the advecting velocity at node p = (i, j, k): a bilinear transpose (kinds
// 2..7), else a field plus a.shift (kind 1) or itself
template <int BIL>
__device__ __forceinline__ double adv_vel(const AdvSrc &a, const Dims &d, long long p, int i, int j, int k)
{
    const double *f = a.a + p;
    if (BIL == ADV_FIELD) return a.kind == 1 ? ad(f[0], a.shift) : f[0];
    double q0 = f[a.off[0]], q1 = f[a.off[1]], q2 = f[a.off[2]], q3 = f[a.off[3]];
    if (a.pin && i == 0) {   // kinds 4 and 6 at the open faces
        if (a.kind == 4 && j > 0) { q0 = a.pin[(long long)k * a.pNY + j - 1]; q2 = a.pin[(long long)k * a.pNY + j]; }
        if (a.kind == 6 && k > 0) { q0 = a.pin[(long long)(k - 1) * a.pNY + j]; q2 = a.pin[(long long)k * a.pNY + j]; }
    }
    if (a.pout && i == a.nx - 1) {
        if (a.kind == 4 && j > 0) { q1 = a.pout[(long long)k * a.pNY + j - 1]; q3 = a.pout[(long long)k * a.pNY + j]; }
        if (a.kind == 6 && k > 0) { q1 = a.pout[(long long)(k - 1) * a.pNY + j]; q3 = a.pout[(long long)k * a.pNY + j]; }
    }
    return interp<BIL>(q0, q1, q2, q3, a, a.ax == 0 ? i : k, a.ay == 1 ? j : k);
}

// D0 of buffer index b (ghost rules precomputed in the table; line = k*NY + j
// of an x line, for the open-face planes)
__device__ __forceinline__ double d0_at(const EnoTab &T, const double *__restrict__ q, long long base,
                                        long long stride, int b, double qf, double ql, long long line = 0)
{
    int r = T.r;
    if (b >= r && b < T.nb - r) return q[base + (long long)(b - r + T.s0) * stride];
    int gi = (b < r) ? b : 3 + (T.nb - 1 - b);
    int src = T.gsrc[gi];
    if (src == 0) return 0.0;
    if (src == 3) return T.glo[line];
    if (src == 4) return T.ghi[line];
    return ml(T.gm[gi], src == 1 ? qf : ql);
}

// the divided differences of a line: UNI, one power-of-two spacing (T.uni)
template <bool UNI>
__device__ __forceinline__ double diff1(const EnoTab &T, double a, int b)
{
    return UNI ? ml(a, T.ru1) : dd(T, a, T.d1[b]);
}
template <bool UNI>
__device__ __forceinline__ double diff2(const EnoTab &T, double a, int b)
{
    return UNI ? ml(a, T.ru2) : dd(T, a, T.d2[b]);
}
template <bool UNI>
__device__ __forceinline__ double diff3(const EnoTab &T, double a, int b)
{
    return UNI ? div_by_spacing_2t(a, T.uh3, T.ru3, T.ru3l) : dd(T, a, T.d3[b]);
}

// d + c g rounded as the product and then the sum, for g a power of two in
// [2^-200, 2^200]: one FMA, unless the product could be subnormal
__device__ __noinline__ double mul_add_call(double c, double g, double d) { return ad(d, ml(c, g)); }
__device__ __forceinline__ double add_scaled(double d, double c, double g)
{
    const DWords w = dwords(c);
    if ((w.hi & 0x7ff00000u) >= 0x0d000000u || dw_zero(w)) return __fma_rn(c, g, d);   // exponent of c >= -815
    return mul_add_call(c, g, d);
}

// ENO_compute_convective_terms body for node c (ENO.c:184-244).  UNI: the
// factors g2 = +-h and g3 = 2h^2, -h^2, 2h^2 are powers of two, so a product
// with them is exact and rounding it with the sum (one FMA) changes nothing
template <int R, bool UNI>
__device__ __forceinline__ double eno_eval(const EnoTab &T, double vel, double d1m1, double d1c, double d2m1, double d2c,
                                          double d2p1, double d3m2, double d3m1, double d3c, double d3p1, int c)
{
    bool up = positive(vel);
    double dQ = up ? d1m1 : d1c;
    if (R > 1) {
        double a = up ? d2m1 : d2c, b = up ? d2c : d2p1;
        bool left = abs_le(a, b);
        double cc = left ? a : b;
        dQ = UNI ? add_scaled(dQ, cc, up ? T.uh : -T.uh) : ad(dQ, ml(cc, T.g2[2 * c + (up ? 0 : 1)]));
        if (R > 2) {
            int kso = (up ? -1 : 0) + (left ? -1 : 0);
            double e = kso == -2 ? d3m2 : (kso == -1 ? d3m1 : d3c);
            double f = kso == -2 ? d3m1 : (kso == -1 ? d3c : d3p1);
            double cs = abs_le(e, f) ? e : f;
            dQ = UNI ? add_scaled(dQ, cs, kso == -1 ? T.ug3m : T.ug3) : ad(dQ, ml(cs, T.g3[3 * c + kso + 2]));
        }
    }
    return ml(vel, dQ);
}

// x pass: one block per line (j = t1, k = t2)
template <int R, bool UNI, int BIL>
__global__ void k_eno_x(Dims d, EnoTab T, const double *__restrict__ q, AdvSrc adv, int t1a, int t2a,
                        int first, double *__restrict__ conv)
{
    extern __shared__ double sm[];
    int nb = T.nb;
    double *s0 = sm, *s1 = sm + nb, *s2 = sm + 2 * nb, *s3 = sm + 3 * nb;
    int j = t1a + blockIdx.x, k = t2a + blockIdx.y;
    long long base = d.at(0, j, k);
    double qf = q[base + T.s0], ql = q[base + T.e0];
    const long long line = (long long)k * T.gNY + j;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) s0[b] = d0_at(T, q, base, 1, b, qf, ql, line);
    __syncthreads();
    for (int b = threadIdx.x; b < nb - 1; b += blockDim.x) s1[b] = diff1<UNI>(T, sb(s0[b + 1], s0[b]), b);
    __syncthreads();
    if (R > 1) {
        for (int b = 1 + threadIdx.x; b < nb - 1; b += blockDim.x) s2[b] = diff2<UNI>(T, sb(s1[b], s1[b - 1]), b);
        __syncthreads();
    }
    if (R > 2) {
        for (int b = 1 + threadIdx.x; b < nb - 2; b += blockDim.x) s3[b] = diff3<UNI>(T, sb(s2[b + 1], s2[b]), b);
        __syncthreads();
    }
    for (int c = R + threadIdx.x; c < nb - R; c += blockDim.x) {
        int i = c - R + T.s0;
        long long p = base + i;
        double vel = adv_vel<BIL>(adv, d, p, i, j, k);
        double o = eno_eval<R, UNI>(T, vel, s1[c - 1], s1[c], R > 1 ? s2[c - 1] : 0.0, R > 1 ? s2[c] : 0.0,
                                    R > 1 ? s2[c + 1] : 0.0, R > 2 ? s3[c - 2] : 0.0, R > 2 ? s3[c - 1] : 0.0,
                                    R > 2 ? s3[c] : 0.0, R > 2 ? s3[c + 1] : 0.0, c);
        conv[p] = first ? o : ad(conv[p], o);
    }
}

// nodes per segment of a y / z line: as many as leave ENO_SEG_THREADS threads,
// at most ENO_SEG_MAX (a segment starts with 15 differences of its own, a
// line's step is 15 to 20 FP64 operations one after the other).  Measured us
// per pass with 1 / 8 / 16 / 32 / 64 nodes: 32x16x16 6.0 / 12.7 / 19 / 19 / 19,
// 128x64x64 52 / 28 / 36 / 58 / 106, 256x128x128 379 / 168 / 157 / 154 / 164
constexpr int ENO_SEG_MAX = 32, ENO_SEG_THREADS = 65536;


// y / z pass: one thread per segment of a line (blockIdx.z of nseg), a
// sliding window along it.  A segment starts its window afresh from the
// buffer entries before it, so every divided difference is formed from the
// same operands as in one walk of the whole line and the results are the same
// bits; the segments multiply the threads in flight, which hide the latency
// of the line walk.
// 16 blocks of 64 per SM (64 registers, a few spilled to L1): measured 3.7 %
// faster at 512x256x256 than the 10 blocks that 96 registers allow, and
// faster than 12, 20 or 24 blocks
template <int R, bool UNI, int BIL>
__global__ void __launch_bounds__(64, 16) k_eno_yz(Dims d, int dir, EnoTab T, const double *__restrict__ q, AdvSrc adv, int t1a,
                         int t1b, int t2a, int first, int seglen, double *__restrict__ conv)
{
    int i = t1a + blockIdx.x * blockDim.x + threadIdx.x;
    if (i > t1b) return;
    int o2 = t2a + blockIdx.y;   // k for the y pass, j for the z pass
    const int cs = R + blockIdx.z * seglen, ce = min(cs + seglen, T.nb - R);
    if (cs >= ce) return;
    long long stride = dir == 1 ? d.PX : d.plane;
    long long base = dir == 1 ? d.at(i, 0, o2) : d.at(i, o2, 0);
    double qf = q[base + (long long)T.s0 * stride], ql = q[base + (long long)T.e0 * stride];
    const int W = 2 * R + 1;
    const int b0 = cs - R;       // buffer index of the window's first entry
    double w0[7], w1[6], w2[5], w3[4];
    // window for c = cs
#pragma unroll
    for (int t = 0; t < W; t++) w0[t] = d0_at(T, q, base, stride, b0 + t, qf, ql);
#pragma unroll
    for (int t = 0; t < 2 * R; t++) w1[t] = diff1<UNI>(T, sb(w0[t + 1], w0[t]), b0 + t);
    if (R > 1) {
#pragma unroll
        for (int t = 0; t < 2 * R - 1; t++) w2[t] = diff2<UNI>(T, sb(w1[t + 1], w1[t]), b0 + t + 1);
    }
    if (R > 2) {
#pragma unroll
        for (int t = 0; t < 2 * R - 2; t++) w3[t] = diff3<UNI>(T, sb(w2[t + 1], w2[t]), b0 + t + 1);
    }
    for (int c = cs; c < ce; c++) {
        int m = c - R + T.s0;
        long long p = base + (long long)m * stride;
        int jj = dir == 1 ? m : o2, kk = dir == 1 ? o2 : m;
        double vel = adv_vel<BIL>(adv, d, p, i, jj, kk);
        constexpr int R2 = R > 1 ? R - 2 : 0;
        double o = eno_eval<R, UNI>(T, vel, w1[R - 1], w1[R], R > 1 ? w2[R2] : 0.0, R > 1 ? w2[R2 + 1] : 0.0,
                                    R > 1 ? w2[R2 + 2] : 0.0, R > 2 ? w3[0] : 0.0, R > 2 ? w3[1] : 0.0,
                                    R > 2 ? w3[2] : 0.0, R > 2 ? w3[3] : 0.0, c);
        conv[p] = first ? o : ad(conv[p], o);
        if (c + 1 < ce) {
            // slide: new D0[c+1+R], D1[c+R], D2[c+R], D3[c+R-1]
#pragma unroll
            for (int t = 0; t < W - 1; t++) w0[t] = w0[t + 1];
            w0[W - 1] = d0_at(T, q, base, stride, c + 1 + R, qf, ql);
#pragma unroll
            for (int t = 0; t < 2 * R - 1; t++) w1[t] = w1[t + 1];
            w1[2 * R - 1] = diff1<UNI>(T, sb(w0[W - 1], w0[W - 2]), c + R);
            if (R > 1) {
#pragma unroll
                for (int t = 0; t < 2 * R - 2; t++) w2[t] = w2[t + 1];
                w2[2 * R - 2] = diff2<UNI>(T, sb(w1[2 * R - 1], w1[2 * R - 2]), c + R);
            }
            if (R > 2) {
#pragma unroll
                for (int t = 0; t < 2 * R - 3; t++) w3[t] = w3[t + 1];
                w3[2 * R - 3] = diff3<UNI>(T, sb(w2[2 * R - 2], w2[2 * R - 3]), c + R - 1);
            }
        }
    }
}

// one full line exactly as ENO.c (host line API)
__global__ void k_eno_line(int order, int n, const double *__restrict__ D0, const double *__restrict__ P,
                           const double *__restrict__ V, double *__restrict__ out)
{
    extern __shared__ double sm[];
    double *D1 = sm, *D2 = sm + n, *D3 = sm + 2 * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) { D1[i] = 0.0; D2[i] = 0.0; D3[i] = 0.0; }
    __syncthreads();
    for (int i = threadIdx.x; i < n - 1; i += blockDim.x) D1[i] = dv(sb(D0[i + 1], D0[i]), sb(P[i + 1], P[i]));
    __syncthreads();
    if (order > 1)
        for (int i = 1 + threadIdx.x; i < n - 1; i += blockDim.x) D2[i] = dv(sb(D1[i], D1[i - 1]), sb(P[i + 1], P[i - 1]));
    __syncthreads();
    if (order > 2)
        for (int i = 1 + threadIdx.x; i < n - 2; i += blockDim.x) D3[i] = dv(sb(D2[i + 1], D2[i]), sb(P[i + 2], P[i - 1]));
    __syncthreads();
    for (int i = order + threadIdx.x; i < n - order; i += blockDim.x) {
        int k = V[i] > 0.0 ? i - 1 : i, ks = 0;
        double dQ = D1[k];
        if (order > 1) {
            double c;
            if (fabs(D2[k]) <= fabs(D2[k + 1])) { c = D2[k]; ks = k - 1; }
            else { c = D2[k + 1]; ks = k; }
            dQ = ad(dQ, ml(c, ad(sb(P[i], P[k]), sb(P[i], P[k + 1]))));
        }
        if (order > 2) {
            double cs = fabs(D3[ks]) <= fabs(D3[ks + 1]) ? D3[ks] : D3[ks + 1];
            double xi = P[i], a = P[ks], b = P[ks + 1], e = P[ks + 2];
            double g = ad(ad(ml(sb(xi, a), sb(xi, b)), ml(sb(xi, b), sb(xi, e))), ml(sb(xi, a), sb(xi, e)));
            dQ = ad(dQ, ml(cs, g));
        }
        out[i] = ml(V[i], dQ);
    }
}

}  // namespace

namespace {
template <int R, bool UNI, int BIL>
void eno_pass(cudaStream_t s, const Dims &d, int dir, const EnoTab &tab, const double *q, const AdvSrc &adv, int t1a,
              int t1b, int t2a, int t2b, int first, double *conv, int segments)
{
    const int n1 = t1b - t1a + 1, n2 = t2b - t2a + 1, ncen = tab.nb - 2 * tab.r;
    if (dir == 0) {
        k_eno_x<R, UNI, BIL><<<dim3(n1, n2), 128, sizeof(double) * 4 * (size_t)tab.nb, s>>>(d, tab, q, adv, t1a, t2a, first, conv);
        return;
    }
    const int want = (int)std::min<long long>(ENO_SEG_MAX, std::max(1ll, (long long)n1 * n2 * ncen / ENO_SEG_THREADS));
    const int nseg = segments > 0 ? segments : std::max(1, (ncen + want / 2) / want);
    const int seglen = (ncen + nseg - 1) / nseg;
    k_eno_yz<R, UNI, BIL><<<dim3((n1 + 63) / 64, n2, nseg), 64, 0, s>>>(d, dir, tab, q, adv, t1a, t1b, t2a, first, seglen, conv);
}
}  // namespace

// segments: per y / z line, 0 = the rule of ENO_SEG_*, 1 = each line walked by
// one thread
void launch_eno_pass(cudaStream_t s, const Dims &d, int dir, const EnoTab &tab, const double *q, AdvSrc adv,
                     int t1a, int t1b, int t2a, int t2b, int first, double *conv, int segments)
{
    if (t1b < t1a || t2b < t2a) return;
    const bool uni = tab.uni && tab.fastdiv, bil = adv.kind >= 2;
    if (bil) {
        const long long X = 1, Y = d.PX, Z = d.plane;
        // kind: lower node of the pair along the first axis, upper one; the
        // second axis adds its step (the order q0 .. q3 of interp4)
        const long long o[6][4] = {{-X, 0, -X + Y, Y}, {-X, 0, -X + Z, Z}, {-Y, -Y + X, 0, X},
                                   {-Y, -Y + Z, 0, Z}, {-Z, -Z + X, 0, X}, {-Z, 0, -Z + Y, Y}};
        const int ax[6] = {0, 0, 0, 2, 0, 2}, ay[6] = {1, 2, 1, 1, 2, 1};
        for (int t = 0; t < 4; t++) adv.off[t] = o[adv.kind - 2][t];
        adv.ax = ax[adv.kind - 2];
        adv.ay = ay[adv.kind - 2];
    }
    auto run = [&](auto pass) { pass(s, d, dir, tab, q, adv, t1a, t1b, t2a, t2b, first, conv, segments); };
    auto order = [&](auto r) {
        constexpr int R = decltype(r)::value;
        auto spacing = [&](auto u) {
            constexpr bool UNI = decltype(u)::value;
            if (!bil) run(eno_pass<R, UNI, ADV_FIELD>);
            else if (!adv.wx.half) run(eno_pass<R, UNI, ADV_BILINEAR>);
            else if (!adv.wy.half) run(eno_pass<R, UNI, ADV_HALF_X>);
            else run(eno_pass<R, UNI, ADV_HALF>);
        };
        if (uni) spacing(std::true_type{});
        else spacing(std::false_type{});
    };
    if (tab.r == 1) order(std::integral_constant<int, 1>{});
    else if (tab.r == 2) order(std::integral_constant<int, 2>{});
    else order(std::integral_constant<int, 3>{});
}

int launch_eno_line(int order, int n, const double *D0, const double *P, const double *V, double *out,
                    cudaStream_t s)
{
    size_t sh = sizeof(double) * 3 * (size_t)n;
    if (sh > 200 * 1024) return 1;
    if (sh > 48 * 1024) cudaFuncSetAttribute(k_eno_line, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
    k_eno_line<<<1, 256, sh, s>>>(order, n, D0, P, V, out);
    return 0;
}
