// k_mglow.cu -- the lower part of the pressure V-cycle in one launch.
//
// A V-cycle visits its coarse levels with up to 24 half sweeps each way, and
// every one of them depends on the one before.  As a kernel per half sweep a
// level of 2^11 .. 2^17 cells costs about 2.2 us per half sweep whatever its
// size (launch, drain, the L2 round trips of its loads), and a single block
// sweeping in global memory needed 2.3 us, although the arithmetic takes a
// tenth of that: latency bounds it.  Here the levels from the first one of at
// most MG_LOW_CELLS32 / MG_LOW_CELLS64 cells down to the coarsest run in one
// thread-block cluster of 16 blocks (8 or 1 where the device cannot hold
// one) with x in shared memory:
//
//  * a level's rows (row = k ny + j) are dealt to the blocks in runs of
//    rpc rows; a block keeps a window of its rows and ny rows either side
//    (the rows j +- 1 and k +- 1 of its own), per colour, with a spare
//    column at each end, so every neighbour is a local load at a fixed
//    distance.  b, 1/diag and the six coefficients of a thread's cells are
//    formed once per visit and stay in registers;
//  * a new value is stored in the own window and pushed into the windows of
//    the (at most four) blocks that read it, then the hardware cluster
//    barrier ends the half sweep (about 1000 cycles with the pushes);
//  * levels of at most MG_LOW_ONE32 / MG_LOW_ONE64 cells are swept by block 0
//    alone, a block barrier per half sweep over the warps that own cells
//    (measured: 130 cycles per half sweep at 256 cells, 670 at 4096);
//  * residuals, right-hand sides and corrections pass between the cluster's
//    levels through the levels' global arrays (L2), between one block's levels
//    through its shared memory.
//
// Every cell's operations are those of the kernels in k_mg.cu, in the same
// order (an absent neighbour has a zero coefficient instead of a skipped
// operation), so the iterates are the same bits.  Measured per V-cycle,
// before and after: 32x16x16 139 -> 63 us, 128x64x64 (x spacing 8 times y's)
// 445 -> 223 us, 256x128x128 stretched 630 -> 421 us, 64x32x32 in FP64 283 ->
// 228 us.  The line at 32768 cells: a 131072-cell level takes 2.3 us per half
// sweep as launches on every SM against 4.5 us on the cluster's 16; a 32768-cell
// one 2.2 us against 0.85 us.  In FP64 (1/64 of the FP32 rate) a level of
// more than 512 cells is faster over the cluster than in one block.
#include <vector>

#include "turb_internal.cuh"
#include "turb_mg.cuh"

namespace {

constexpr int LOW_THREADS = 512;

// cells per thread and colour a level may have: b and 1/diag live in registers
template <typename T> struct Low;
template <> struct Low<float> { static constexpr int CPT = 4; };
template <> struct Low<double> { static constexpr int CPT = 2; };

template <typename T>
struct alignas(16) LowRow {
    T dy, dz, rs, rn, rb, rf;   // widths, 1/face distance to the four row neighbours (0: absent)
    int par;                    // (j + k) & 1
    unsigned mask;              // blocks of the cluster whose window holds the row
};

template <typename T>
struct LowLev {
    MgDevLevel L;
    T *x, *b, *r;
    const T *invd;
    int pre, post;
    int ctas, rows, rpc, hx, pitch;
    // byte offsets in shared memory: x windows, row table, 1/diag of the own
    // cells (by colour and pair), the level's packed tables (LowTab); on a
    // level that one block sweeps also its residual, and its b where the finer
    // level is such a level too (bsm)
    unsigned xoff, roff, ioff, toff, eoff, boff;
    int bsm;
};

// A level's 1-D tables as mg_low_tables packs them: widths and 1/face
// distances (0 where the face is absent), along x split by parity of i, and
// the transfer tables of Xfer1D per direction
template <typename T>
struct LowTab {
    const T *col;                         // dx, 1/f left, 1/f right: [3][2][hx]
    const T *ry, *rz;                     // [3][ny], [3][nz]
    const T *w0[3], *w1[3], *rw[3];
    const int *I0[3], *I1[3], *rf[3];
    __device__ __forceinline__ LowTab(const unsigned char *p, const MgDevLevel &F, const MgDevLevel &C, int hx)
    {
        const int nf[3] = {F.nx, F.ny, F.nz}, nc[3] = {C.nx, C.ny, C.nz};
        const T *t = reinterpret_cast<const T *>(p);
        col = t;
        t += 6 * hx;
        ry = t;
        rz = t + 3 * F.ny;
        t += 3 * (F.ny + F.nz);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            w0[a] = t;
            w1[a] = t + nf[a];
            rw[a] = t + 2 * nf[a];
            t += 2 * nf[a] + 4 * nc[a];
        }
        const int *i = reinterpret_cast<const int *>(t);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            I0[a] = i;
            I1[a] = i + nf[a];
            rf[a] = i + 2 * nf[a];
            i += 2 * nf[a] + 4 * nc[a];
        }
    }
};
template <typename T>
__host__ __device__ inline unsigned low_tab_bytes(const MgDevLevel &F, const MgDevLevel &C)
{
    const unsigned n = 2u * (F.nx + F.ny + F.nz) + 4u * (C.nx + C.ny + C.nz), hx = (F.nx + 1) / 2;
    return ((6u * hx + 3u * (F.ny + F.nz) + n) * (unsigned)sizeof(T) + n * 4u + 15u) & ~15u;
}

template <typename T>
struct LowArgs {
    int nlev, ctas;
    unsigned zero_bytes, inv_off, xl_off;   // xl: x of the coarsest level
    const double *coarse_inv;
    LowLev<T> v[MG_LOW_MAXLEV];
};

__device__ __forceinline__ float lmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double lmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float ladd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double ladd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float lfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double lfma(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ void cluster_bar()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void push(uint32_t addr, unsigned rank, float v)
{
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}
__device__ __forceinline__ void push(uint32_t addr, unsigned rank, double v)
{
    uint32_t ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}

extern __shared__ __align__(16) unsigned char low_sm[];

template <int BYTES>
__device__ __forceinline__ void copy_async(void *smem, const void *gmem)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(a), "l"(gmem), "n"(BYTES) : "memory");
}

// storage index of cell (i, row) of a level; par = (j + k) & 1
__device__ __forceinline__ int cell_at(const MgDevLevel &L, int i, int row, int par)
{
    const int c = row * L.nx + i;
    return L.split ? (((i + par) & 1) * ((L.nx * L.ny * L.nz) >> 1) + (c >> 1)) : c;
}

// One level as a block sees it: its run of rows, its windows in shared memory
// (indices in units of T from its base) and its cells
template <typename T>
struct Lev {
    int nx, ny, hx, pitch, wsz, rpc, r0, nloc, xo, co, ro, io, dr, dm, rl0, m0;

    __device__ __forceinline__ void open(const LowLev<T> &v, int rank)
    {
        nx = v.L.nx;
        ny = v.L.ny;
        hx = v.hx;
        pitch = v.pitch;
        rpc = v.rpc;
        wsz = (rpc + 2 * ny) * pitch;
        r0 = rank * rpc;
        nloc = max(0, min(rpc, v.rows - r0)) * hx;
        xo = (int)(v.xoff / sizeof(T));
        co = (int)(v.toff / sizeof(T));
        ro = (int)v.roff;
        io = (int)(v.ioff / sizeof(T));
        dr = LOW_THREADS / hx;
        dm = LOW_THREADS - dr * hx;
        rl0 = (int)threadIdx.x / hx;
        m0 = (int)threadIdx.x - rl0 * hx;
    }
    // the block's cell pair q of this thread (i = 2 m and 2 m + 1 of own row rl)
    __device__ __forceinline__ bool has(int q) const { return q * LOW_THREADS + (int)threadIdx.x < nloc; }
    // the next pair of the thread after (rl, m)
    __device__ __forceinline__ void next(int &rl, int &m) const
    {
        rl += dr;
        m += dm;
        if (m >= hx) {
            m -= hx;
            rl++;
        }
    }
    __device__ __forceinline__ int at(int rl, int m) const { return (rl + ny) * pitch + m + 1; }
    __device__ __forceinline__ const LowRow<T> &row(int rl) const
    {
        return *reinterpret_cast<const LowRow<T> *>(low_sm + ro + rl * (int)sizeof(LowRow<T>));
    }
    // the six neighbour coefficients of cell 2 m + p
    __device__ __forceinline__ void coef(const LowRow<T> &R, int m, int p, T (&f)[6]) const
    {
        const T *c = reinterpret_cast<const T *>(low_sm) + co + p * hx + m;
        const T dx = c[0], rl = c[2 * hx], rr = c[4 * hx];
        const T dyz = lmul(R.dy, R.dz), dxz = lmul(dx, R.dz), dxy = lmul(dx, R.dy);
        f[0] = lmul(dyz, rl);
        f[1] = lmul(dyz, rr);
        f[2] = lmul(dxz, R.rs);
        f[3] = lmul(dxz, R.rn);
        f[4] = lmul(dxy, R.rb);
        f[5] = lmul(dxy, R.rf);
    }
    // sum f x_nb over the neighbours (the other colour's window, w its index
    // of the west one, s of the cell itself)
    __device__ __forceinline__ T gather(const T *S, int w, int s, const T (&f)[6]) const
    {
        const int np = ny * pitch;
        const T xw = S[w], xe = S[w + 1], xs = S[s - pitch], xn = S[s + pitch], xb = S[s - np], xf = S[s + np];
        T a = lfma(f[0], xw, T(0));
        a = lfma(f[1], xe, a);
        a = lfma(f[2], xs, a);
        a = lfma(f[3], xn, a);
        a = lfma(f[4], xb, a);
        return lfma(f[5], xf, a);
    }
    // a new value into the windows of the other blocks that read the row
    __device__ __forceinline__ void push_all(T *S, int idx, unsigned mask, T val) const
    {
        const int rank = r0 / rpc;
        while (mask) {
            const int t = __ffs(mask) - 1;
            mask &= mask - 1;
            push(static_cast<uint32_t>(__cvta_generic_to_shared(S + (idx + (rank - t) * rpc * pitch))), t, val);
        }
    }
};

// A thread's cells of one colour.  A pair that has no cell of the colour (odd
// row ends, threads past the block's rows) stands for the spare column of the
// window's first own row with b, 1/diag and the coefficients zero: it reads
// and writes zeros there, and the sweeps need no test
template <typename T, int Q>
struct Cells {
    T b[Q], iv[Q];
    T f[Q][6];        // neighbour coefficients
    int s[Q], w[Q];   // the cell in its colour's window; its west neighbour in the other's
};

// The cells of a level in the order their colours are swept; b from the
// level's array.  far: the blocks that read the pair's row
template <typename T, int Q>
__device__ __forceinline__ void low_load(const Lev<T> &V, const LowLev<T> &v, int c0, Cells<T, Q> (&c)[2], unsigned (&far)[Q])
{
    const MgDevLevel &L = v.L;
    const T *S = reinterpret_cast<const T *>(low_sm);
    const int base[2] = {V.xo + c0 * V.wsz, V.xo + (1 - c0) * V.wsz}, np = v.rpc * V.hx;
    const int spare = V.ny * V.pitch, bs = (int)(v.boff / sizeof(T));
    int rl = V.rl0, m = V.m0;
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const bool has = V.has(q);
        const int r = has ? rl : 0, i2 = has ? m : 0, t = has ? q * LOW_THREADS + (int)threadIdx.x : 0;
        const LowRow<T> R = V.row(r);
        far[q] = has ? R.mask : 0u;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int p = (R.par + c0 + h) & 1;
            const bool k = has && 2 * i2 + p < V.nx;
            T b = v.bsm ? S[bs + (c0 ^ h) * np + t] : __ldcg(v.b + (k ? cell_at(L, 2 * i2 + p, V.r0 + r, R.par) : 0));
            T f[6];
            V.coef(R, i2, p, f);
            c[h].b[q] = k ? b : T(0);
            c[h].iv[q] = k ? S[V.io + (c0 ^ h) * np + t] : T(0);
            c[h].s[q] = base[h] + (k ? V.at(r, i2) : spare);
            c[h].w[q] = base[1 - h] + (k ? V.at(r, i2) - 1 + p : spare);
#pragma unroll
            for (int e = 0; e < 6; e++) c[h].f[q][e] = k ? f[e] : T(0);
        }
        V.next(rl, m);
    }
}

// one half sweep; o: distance from a window to the other colour's
template <typename T, int Q, bool CL, bool ZERO>
__device__ __forceinline__ void low_half(const Lev<T> &V, const Cells<T, Q> &c, int o, const unsigned (&far)[Q])
{
    T *S = reinterpret_cast<T *>(low_sm);
    T val[Q];
#pragma unroll
    for (int q = 0; q < Q; q++)
        val[q] = ZERO ? lmul(c.b[q], c.iv[q]) : lmul(ladd(c.b[q], V.gather(S, c.w[q], c.s[q] + o, c.f[q])), c.iv[q]);
#pragma unroll
    for (int q = 0; q < Q; q++) {
        S[c.s[q]] = val[q];
        if (CL && far[q]) V.push_all(S, c.s[q], far[q], val[q]);
    }
}

template <bool CL>
__device__ __forceinline__ void low_bar(int act)
{
    if (CL) cluster_bar();
    else asm volatile("bar.sync 1, %0;" ::"r"(act) : "memory");
}

// n sweeps (from x = 0 if ZERO), a barrier after each half sweep.  CL: the
// whole cluster sweeps; else the warps of one block that own cells
template <typename T, int Q, bool CL, bool ZERO>
__device__ __forceinline__ void low_sweeps(const Lev<T> &V, const Cells<T, Q> (&c)[2], int o, const unsigned (&far)[Q], int n)
{
    const int act = min(LOW_THREADS, (V.nloc + 31) / 32 * 32);
    if (CL || (int)threadIdx.x < act) {
        if (ZERO) {
            low_half<T, Q, CL, true>(V, c[0], o, far);
            low_bar<CL>(act);
            low_half<T, Q, CL, false>(V, c[1], -o, far);
            low_bar<CL>(act);
        }
#pragma unroll 1
        for (int it = ZERO ? 1 : 0; it < n; it++) {
            low_half<T, Q, CL, false>(V, c[0], o, far);
            low_bar<CL>(act);
            low_half<T, Q, CL, false>(V, c[1], -o, far);
            low_bar<CL>(act);
        }
    }
    if (!CL) __syncthreads();
}

// the sweeps of a level: down from x = 0, up with the colours reversed
template <typename T, int Q, bool CL>
__device__ __noinline__ void low_smooth(const LowLev<T> &v, int rank, bool down)
{
    Lev<T> V;
    V.open(v, rank);
    Cells<T, Q> c[2];
    unsigned far[Q];
    low_load<T, Q>(V, v, down ? 0 : 1, c, far);
    if (down) low_sweeps<T, Q, CL, true>(V, c, V.wsz, far, v.pre);
    else low_sweeps<T, Q, CL, false>(V, c, -V.wsz, far, v.post);
}

// What a level does once per visit is kept in small loops, shared by all
// levels: straight-line code runs at the speed of the instruction fetch here.

// residual r = b - S x (natural order)
template <typename T>
__device__ __noinline__ void low_resid(const LowLev<T> &v, int rank)
{
    Lev<T> V;
    V.open(v, rank);
    const T *S = reinterpret_cast<const T *>(low_sm);
    const T pin = (T)v.L.pin;
    T *r = v.r, *E = reinterpret_cast<T *>(low_sm) + v.eoff / sizeof(T);
    const int np = v.rpc * V.hx, bs = (int)(v.boff / sizeof(T));
    int rl = V.rl0, m = V.m0;
#pragma unroll 1
    for (int t = threadIdx.x; t < V.nloc; t += LOW_THREADS, V.next(rl, m)) {
        const LowRow<T> R = V.row(rl);
        const int g = V.r0 + rl, s = V.at(rl, m);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int p = (R.par + h) & 1, i = 2 * m + p, x = V.xo + h * V.wsz, o = V.xo + (1 - h) * V.wsz;
            if (i >= V.nx) continue;
            const T b = v.bsm ? S[bs + h * np + t] : __ldcg(v.b + cell_at(v.L, i, g, R.par));
            T f[6];
            V.coef(R, m, p, f);
            const T off = V.gather(S, o + s - 1 + p, o + s, f);
            T dg = ladd(ladd(ladd(ladd(ladd(f[0], f[1]), f[2]), f[3]), f[4]), f[5]);
            if (i == V.nx - 1 && g == v.rows - 1) dg = ladd(dg, pin);
            const T res = ladd(b, -lfma(dg, S[x + s], -off));
            if (v.ctas > 1) __stcg(r + g * V.nx + i, res);
            else E[g * V.nx + i] = res;
        }
    }
}

// x + the linear prolongation of the coarser level's x; xl >= 0: that is the
// coarsest level, its x at index xl of shared memory (block 0)
template <typename T>
__device__ __noinline__ void low_prolong(const LowLev<T> &v, const LowLev<T> &vc, int xl, int rank)
{
    Lev<T> V;
    V.open(v, rank);
    const MgDevLevel &C = vc.L;
    const LowTab<T> X(low_sm + v.toff, v.L, C, v.hx);
    const T *xc = vc.x;
    T *S = reinterpret_cast<T *>(low_sm);
    const bool one = v.ctas == 1;   // the coarser level's x is in this block's shared memory
    const int cxo = (int)(vc.xoff / sizeof(T)), cpitch = vc.pitch, cws = (vc.rpc + 2 * C.ny) * cpitch;
    const int cnx = C.nx, cny = C.ny, half = (C.nx * C.ny * C.nz) >> 1, split = C.split;
    int rl = V.rl0, m = V.m0;
#pragma unroll 1
    for (int t = threadIdx.x; t < V.nloc; t += LOW_THREADS, V.next(rl, m)) {
        const LowRow<T> R = V.row(rl);
        const int g = V.r0 + rl, k = g / V.ny, j = g - k * V.ny, s = V.at(rl, m);
        const int Jy[2] = {X.I0[1][j], X.I1[1][j]}, Kz[2] = {X.I0[2][k], X.I1[2][k]};
        T val[2][8];
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int i = min(2 * m + p, V.nx - 1);
            const int Ix[2] = {X.I0[0][i], X.I1[0][i]};
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const int J = Jy[(e >> 1) & 1], K = Kz[e >> 2], I = Ix[e & 1], g2 = K * cny + J, at = g2 * cnx + I;
                const int cc = (I + J + K) & 1;
                if (!one) val[p][e] = __ldcg(xc + (split ? cc * half + (at >> 1) : at));
                else val[p][e] = S[xl >= 0 ? xl + at : cxo + cc * cws + (g2 + cny) * cpitch + (I >> 1) + 1];
            }
        }
#pragma unroll
        for (int p = 0; p < 2; p++) {
            const int i = 2 * m + p, x = V.xo + ((p + R.par) & 1) * V.wsz + s;
            if (i >= V.nx) continue;
            T acc = mg_prolong8<T>(val[p], X.w0[0][i], X.w1[0][i], X.w0[1][j], X.w1[1][j], X.w0[2][k], X.w1[2][k]);
            acc = ladd(S[x], acc);
            S[x] = acc;
            if (R.mask) V.push_all(S, x, R.mask, acc);
        }
    }
}

// x to the level's array
template <typename T>
__device__ __noinline__ void low_store(const LowLev<T> &v, int rank)
{
    Lev<T> V;
    V.open(v, rank);
    const T *S = reinterpret_cast<const T *>(low_sm);
    int rl = V.rl0, m = V.m0;
#pragma unroll 1
    for (int t = threadIdx.x; t < V.nloc; t += LOW_THREADS, V.next(rl, m)) {
        const int par = V.row(rl).par, s = V.at(rl, m);
#pragma unroll
        for (int p = 0; p < 2; p++)
            if (2 * m + p < V.nx)
                __stcg(v.x + cell_at(v.L, 2 * m + p, V.r0 + rl, par), S[V.xo + ((p + par) & 1) * V.wsz + s]);
    }
}

// restriction (the transpose of the prolongation): every block that swept the
// finer level gathers its share of the coarser one's right-hand sides into
// the level's array.  The lists are padded with weight 0 to four entries per
// direction, so the loads are independent
template <typename T>
__device__ __noinline__ void low_restrict(const LowLev<T> &v, const LowLev<T> &vc, double *bl, int rank)
{
    const MgDevLevel &F = v.L, &C = vc.L;
    const LowTab<T> X(low_sm + v.toff, F, C, v.hx);
    const bool one = v.ctas == 1;
    const T *rf = v.r, *E = reinterpret_cast<const T *>(low_sm) + v.eoff / sizeof(T);
    T *b = vc.b, *bs = reinterpret_cast<T *>(low_sm) + vc.boff / sizeof(T);
    const int np = vc.rpc * vc.hx, chx = vc.hx;
    auto at = [&](int o) { return one ? E[o] : __ldcg(rf + o); };
    const int cnx = C.nx, cny = C.ny, nc = C.nx * C.ny * C.nz, half = nc >> 1, split = C.split;
    const int fnx = F.nx, fny = F.ny, step = v.ctas * LOW_THREADS;
    const bool cx = cnx != fnx;   // else one entry of weight 1 along x
    for (int t = rank * LOW_THREADS + (int)threadIdx.x; t < nc; t += step) {
        const int g = t / cnx, I = t - g * cnx, K = g / cny, J = g - K * cny;
        const int *ix = X.rf[0] + 4 * I, *iy = X.rf[1] + 4 * J, *iz = X.rf[2] + 4 * K;
        const T *wx = X.rw[0] + 4 * I, *wy = X.rw[1] + 4 * J, *wz = X.rw[2] + 4 * K;
        T s = 0;
#pragma unroll 1
        for (int h = 0; h < 4; h++) {
            T val[4][4];
#pragma unroll
            for (int d = 0; d < 4; d++)
#pragma unroll
                for (int f = 0; f < 4; f++)
                    if (f == 0 || cx) val[d][f] = at((iz[h] * fny + iy[d]) * fnx + ix[f]);
            s = mg_restrict16<T>(s, val, wz[h], wy, wx, cx);
        }
        if (!one) __stcg(b + (split ? ((I + J + K) & 1) * half + (t >> 1) : t), s);
        else if (bl) bl[t] = (double)s;
        else bs[((I + J + K) & 1) * np + g * chx + (I >> 1)] = s;
    }
}

template <typename T>
__device__ __forceinline__ void low_level_bar(const LowLev<T> &v)
{
    if (v.ctas > 1) cluster_bar();
    else __syncthreads();
}

template <typename T>
__device__ __forceinline__ void low_visit(const LowLev<T> &v, int rank, bool down)
{
    const int q = (v.rpc * v.hx + LOW_THREADS - 1) / LOW_THREADS;   // cell pairs per thread
    if (v.ctas > 1) {
        if (q <= 1) low_smooth<T, 1, true>(v, rank, down);
        else if (q <= 2) low_smooth<T, 2, true>(v, rank, down);
        else low_smooth<T, Low<T>::CPT, true>(v, rank, down);
    } else {
        if (q <= 1) low_smooth<T, 1, false>(v, rank, down);
        else if (q <= 2) low_smooth<T, 2, false>(v, rank, down);
        else low_smooth<T, Low<T>::CPT, false>(v, rank, down);
    }
}

template <typename T>
__global__ void __launch_bounds__(LOW_THREADS, 1) k_vcycle_low(const __grid_constant__ LowArgs<T> arg)
{
    // a copy that the functions below read many times, as words: shared
    // variables cannot have the initialisers of LowArgs' members
    __shared__ __align__(16) unsigned args_sm[sizeof(LowArgs<T>) / 4];
    for (int t = threadIdx.x; t < (int)(sizeof(LowArgs<T>) / 4); t += LOW_THREADS)
        args_sm[t] = reinterpret_cast<const unsigned *>(&arg)[t];
    const LowArgs<T> &a = *reinterpret_cast<const LowArgs<T> *>(args_sm);
    __syncthreads();
    unsigned char *const sm = low_sm;
    pdl_trigger();
    const int tid = threadIdx.x, rank = blockIdx.x, last = a.nlev - 1;
    // the windows start at zero (spare columns and rows outside the level
    // stay so) and the tables are built while the kernel before this one
    // still runs: they depend on the grid only
    for (unsigned t = tid; t < a.zero_bytes / 16; t += LOW_THREADS) reinterpret_cast<uint4 *>(sm)[t] = make_uint4(0, 0, 0, 0);
    for (int l = 0; l < last; l++) {
        const LowLev<T> &v = a.v[l];
        if (rank >= v.ctas) continue;
        const MgDevLevel &L = v.L;
        T *iv = reinterpret_cast<T *>(sm + v.ioff);
        const unsigned char *src = sizeof(T) == 4 ? L.lowf : L.lowd;
        const unsigned nt = low_tab_bytes<T>(L, a.v[l + 1].L);
        for (unsigned t = 16 * tid; t < nt; t += 16 * LOW_THREADS) copy_async<16>(sm + v.toff + t, src + t);
        for (int t = tid; t < v.rpc * v.hx; t += LOW_THREADS) {
            const int rl = t / v.hx, m = t - rl * v.hx, g = rank * v.rpc + rl, k = g / L.ny, par = (g - k * L.ny + k) & 1;
            if (g >= v.rows) break;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int i = 2 * m + ((c + par) & 1);
                if (i < L.nx) copy_async<(int)sizeof(T)>(iv + c * v.rpc * v.hx + t, v.invd + cell_at(L, i, g, par));
            }
        }
    }
    const int ncoarse = a.v[last].L.nx * a.v[last].L.ny * a.v[last].L.nz;
    const int ninv = ncoarse <= MG_LOW_INV ? ncoarse * ncoarse : 0;
    double *inv = reinterpret_cast<double *>(sm + a.inv_off);   // [column][row] where it fits, then the coarsest b
    if (rank == 0)
        for (int t = tid; t < ninv; t += LOW_THREADS) inv[(t % ncoarse) * ncoarse + t / ncoarse] = a.coarse_inv[t];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int l = 0; l < last; l++) {
        const LowLev<T> &v = a.v[l];
        if (rank >= v.ctas) continue;
        const int ny = v.L.ny, nz = v.L.nz;
        const LowTab<T> X(sm + v.toff, v.L, a.v[l + 1].L, v.hx);
        LowRow<T> *row = reinterpret_cast<LowRow<T> *>(sm + v.roff);
        for (int t = tid; t < v.rpc; t += LOW_THREADS) {
            const int g = rank * v.rpc + t;
            if (g >= v.rows) break;
            const int k = g / ny, j = g - k * ny;
            LowRow<T> R;
            R.dy = X.ry[j];
            R.rs = X.ry[ny + j];
            R.rn = X.ry[2 * ny + j];
            R.dz = X.rz[k];
            R.rb = X.rz[nz + k];
            R.rf = X.rz[2 * nz + k];
            R.par = (j + k) & 1;
            R.mask = 0;
            if (v.ctas > 1) {
                if (j > 0) R.mask |= 1u << ((g - 1) / v.rpc);
                if (j < ny - 1) R.mask |= 1u << ((g + 1) / v.rpc);
                if (k > 0) R.mask |= 1u << ((g - ny) / v.rpc);
                if (k < nz - 1) R.mask |= 1u << ((g + ny) / v.rpc);
                R.mask &= ~(1u << rank);
            }
            row[t] = R;
        }
    }
    pdl_wait();
    if (a.ctas > 1) cluster_bar();
    else __syncthreads();

#pragma unroll 1
    for (int l = 0; l < last; l++) {
        const LowLev<T> &v = a.v[l];
        if (rank >= v.ctas) break;
        low_visit<T>(v, rank, true);
        low_resid<T>(v, rank);
        low_level_bar<T>(v);
        low_restrict<T>(v, a.v[l + 1], l + 1 == last ? inv + ninv : nullptr, rank);
        low_level_bar<T>(v);
    }
    if (rank == 0) {   // the coarsest level: its dense inverse
        T *xl = reinterpret_cast<T *>(sm + a.xl_off);
        if (a.v[last - 1].ctas > 1) {
            for (int c = tid; c < ncoarse; c += LOW_THREADS) inv[ninv + c] = (double)__ldcg(a.v[last].b + c);
            __syncthreads();
        }
        for (int r = tid; r < ncoarse; r += LOW_THREADS) {
            double s = 0.0;
            if (ninv)
                for (int c = 0; c < ncoarse; c++) s = __fma_rn(inv[c * ncoarse + r], inv[ninv + c], s);
            else
                for (int c = 0; c < ncoarse; c++) s = __fma_rn(a.coarse_inv[r * ncoarse + c], inv[c], s);
            xl[r] = (T)s;
            __stcg(a.v[last].x + r, (T)s);
        }
    }
    if (rank == 0) __syncthreads();
#pragma unroll 1
    for (int l = last - 1; l >= 0; l--) {
        const LowLev<T> &v = a.v[l];
        if (rank >= v.ctas) continue;
        if (v.ctas > 1 && a.v[l + 1].ctas == 1) cluster_bar();   // block 0 has finished the coarser levels
        low_prolong<T>(v, a.v[l + 1], l + 1 == last ? (int)(a.xl_off / sizeof(T)) : -1, rank);
        low_level_bar<T>(v);
        low_visit<T>(v, rank, false);
        low_store<T>(v, rank);
        // its x is read by the finer level's prolongation, and no block may
        // leave while another still pushes into its windows
        low_level_bar<T>(v);
    }
}

constexpr unsigned align16(unsigned v) { return (v + 15u) & ~15u; }

// the launch's levels, split over the blocks and laid out in shared memory;
// 0 when level l0 and below do not fit, else the dynamic shared memory bytes
template <typename T>
unsigned low_plan(const MgHier<T> &H, int l0, int ctas, LowArgs<T> &a)
{
    a.nlev = H.nl - l0;
    if (a.nlev < 2 || a.nlev > MG_LOW_MAXLEV) return 0;
    a.ctas = 1;
    a.coarse_inv = H.coarse_inv;
    unsigned off = 0;
    for (int t = 0; t < a.nlev; t++) {
        LowLev<T> &v = a.v[t];
        v.L = H.lev[l0 + t];
        v.x = H.x[l0 + t];
        v.b = H.b[l0 + t];
        v.r = H.r[l0 + t];
        v.invd = H.invd[l0 + t];
        const long long n = (long long)v.L.nx * v.L.ny * v.L.nz;
        v.ctas = n > (sizeof(T) == 4 ? MG_LOW_ONE32 : MG_LOW_ONE64) && t + 1 < a.nlev ? ctas : 1;
        v.rows = v.L.ny * v.L.nz;
        v.rpc = (v.rows + v.ctas - 1) / v.ctas;
        v.hx = (v.L.nx + 1) / 2;
        v.pitch = v.hx + 2;
        if (t + 1 == a.nlev) break;
        if ((long long)v.rpc * v.hx > (long long)Low<T>::CPT * LOW_THREADS || v.rpc >= 32768 || v.hx >= 65536) return 0;
        if (v.ctas > a.ctas) a.ctas = v.ctas;
        v.xoff = off;
        off = align16(off + 2u * (v.rpc + 2 * v.L.ny) * v.pitch * (unsigned)sizeof(T));
        if (off > MG_LOW_SMEM) return 0;
    }
    a.zero_bytes = off;
    for (int t = 0; t + 1 < a.nlev; t++) {
        LowLev<T> &v = a.v[t];
        v.roff = off;
        off = align16(off + v.rpc * (unsigned)sizeof(LowRow<T>));
        v.ioff = off;
        off = align16(off + 2u * v.rpc * v.hx * (unsigned)sizeof(T));
        v.toff = off;
        off += low_tab_bytes<T>(v.L, a.v[t + 1].L);
        v.eoff = v.boff = off;
        v.bsm = t > 0 && a.v[t - 1].ctas == 1;
        if (v.ctas == 1) off = align16(off + (unsigned)(v.rows * v.L.nx) * (unsigned)sizeof(T));
        if (v.bsm) {
            v.boff = off;
            off = align16(off + 2u * v.rpc * v.hx * (unsigned)sizeof(T));
        }
    }
    const MgDevLevel &C = a.v[a.nlev - 1].L;
    const unsigned nc = C.nx * C.ny * C.nz;
    a.inv_off = off;
    if (nc > 4096) return 0;
    off += ((nc <= MG_LOW_INV ? nc * nc : 0) + nc) * (unsigned)sizeof(double);
    a.xl_off = off;
    off = align16(off + nc * (unsigned)sizeof(T));
    return off <= MG_LOW_SMEM ? off : 0;
}

template <typename T>
void low_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int ctas, unsigned smem, int pdl)
{
    cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(LOW_THREADS);
    cfg.dynamicSmemBytes = smem;
    int n = 0;
    if (ctas > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)ctas;
        at[n].val.clusterDim.y = 1;
        at[n].val.clusterDim.z = 1;
        n++;
    }
    if (pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
}

}  // namespace

// blocks of the cluster: the most of 16, 8 and 1 that the device holds with
// the largest shared memory a plan may take
template <typename T>
int mg_low_ctas()
{
    if (cudaFuncSetAttribute(k_vcycle_low<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_LOW_SMEM) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (cudaFuncSetAttribute(k_vcycle_low<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) cudaGetLastError();
    for (int ctas = 16; ctas >= 8; ctas /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        low_config<T>(cfg, at, ctas, MG_LOW_SMEM, 0);
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, k_vcycle_low<T>, &cfg) == cudaSuccess && nc >= 1) return ctas;
        cudaGetLastError();
    }
    return 1;
}

template <typename T>
std::vector<unsigned char> mg_low_tables(const MgDevLevel &F, const MgDevLevel &C, const std::vector<T> (&dd)[3],
                                         const std::vector<T> (&rf)[3], const MgXferHost (&x)[3])
{
    const int hx = (F.nx + 1) / 2;
    std::vector<unsigned char> out(low_tab_bytes<T>(F, C), 0);
    T *t = reinterpret_cast<T *>(out.data());
    for (int e = 0; e < 2 * hx; e++) {
        const int p = e >= hx, i = 2 * (e - p * hx) + p;
        if (i >= F.nx) continue;
        t[e] = dd[0][i];
        t[2 * hx + e] = i > 0 ? rf[0][i] : T(0);
        t[4 * hx + e] = i < F.nx - 1 ? rf[0][i + 1] : T(0);
    }
    t += 6 * hx;
    for (int a = 1; a < 3; a++) {
        const int n = a == 1 ? F.ny : F.nz;
        for (int j = 0; j < n; j++) {
            t[j] = dd[a][j];
            t[n + j] = j > 0 ? rf[a][j] : T(0);
            t[2 * n + j] = j < n - 1 ? rf[a][j + 1] : T(0);
        }
        t += 3 * n;
    }
    for (const MgXferHost &d : x) {
        for (double w : d.w0) *t++ = (T)w;
        for (double w : d.w1) *t++ = (T)w;
        for (double w : d.rw) *t++ = (T)w;
    }
    int *i = reinterpret_cast<int *>(t);
    for (const MgXferHost &d : x) {
        for (int v : d.I0) *i++ = v;
        for (int v : d.I1) *i++ = v;
        for (int v : d.rf) *i++ = v;
    }
    return out;
}
template std::vector<unsigned char> mg_low_tables<float>(const MgDevLevel &, const MgDevLevel &, const std::vector<float> (&)[3],
    const std::vector<float> (&)[3], const MgXferHost (&)[3]);
template std::vector<unsigned char> mg_low_tables<double>(const MgDevLevel &, const MgDevLevel &, const std::vector<double> (&)[3],
    const std::vector<double> (&)[3], const MgXferHost (&)[3]);

template <typename T>
int mg_low_fits(const MgHier<T> &H, int l)
{
    LowArgs<T> a;
    return H.low_ctas > 0 && low_plan<T>(H, l, H.low_ctas, a) > 0;
}

template <typename T>
int mg_low(cudaStream_t s, const MgHier<T> &H, int l, const int *pre, const int *post)
{
    LowArgs<T> a;
    const unsigned smem = H.low_ctas > 0 ? low_plan<T>(H, l, H.low_ctas, a) : 0;
    if (!smem) return 0;
    for (int t = 0; t < a.nlev; t++) {
        a.v[t].pre = pre[l + t];
        a.v[t].post = post[l + t];
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    low_config<T>(cfg, at, a.ctas, smem, H.pdl);
    cfg.stream = s;
    cudaLaunchKernelEx(&cfg, k_vcycle_low<T>, a);
    return 1;
}

template int mg_low_ctas<float>();
template int mg_low_ctas<double>();
template int mg_low_fits<float>(const MgHier<float> &, int);
template int mg_low_fits<double>(const MgHier<double> &, int);
template int mg_low<float>(cudaStream_t, const MgHier<float> &, int, const int *, const int *);
template int mg_low<double>(cudaStream_t, const MgHier<double> &, int, const int *, const int *);
