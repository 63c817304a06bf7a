// k_coarse.cu -- the V-cycle's small levels in one launch.
//
// Below some ten thousand cells a smoothing step is a launch with next to no
// work: 2.5 to 4 us each (6 us for lines), seven or more per level.  Here one
// thread-block cluster (16 blocks of 512 threads, one per SM) runs everything
// from the first level that gives each thread at most one cell (8192 cells;
// one segment of the line smoother, 65536 cells) down to the dense coarsest
// solve and back up.  The levels live in the blocks' shared memory: each block
// owns a contiguous share of a level's cells (operator, right-hand side, two
// iterates), a thread keeps its cell in registers while it smooths, and
// neighbours in other blocks are read through distributed shared memory, with
// the cluster's hardware barrier between steps.  Levels too small for that
// belong to the first block alone, which runs them between block barriers
// while the others wait.  The arithmetic is scf_cheb.cuh's and the order of
// every sum that of the one-level kernels, so the result has their bits.
//
// Bound: the latency of a step -- six remote shared-memory reads per cell
// (some 10 cycles per warp and read at an SM's port) and the cluster barrier
// (480 cycles at 512 threads), 1200 to 1800 cycles together.  Measured, a
// whole projection with a launch per step -> with this kernel: 40^3 FP32
// V-cycle 1245 -> 1036 us, 64^3 FP64 2612 -> 2435, 147x93x121 3997 -> 3833,
// 256x128x128 with lines 8677 -> 7465 (the kernel itself 22 us, 27, 21, 119).
// Four cells per thread (32^3 levels) lose: 4000 to 6000 cycles a step where
// the chip-wide kernel takes 2.5 us.  Nor does a cheaper exchange help: with
// the iterates in global memory a step took as long as a launch, and reading
// the block's own cells by plain loads cost more in branches than it saved.
#include "scf_cheb.cuh"
#include "scf_kernels.h"
#include "scf_launch.cuh"

namespace {

constexpr int CC_THREADS = 512, CC_BLOCKS = 16, CC_LEVELS = 12;
constexpr size_t CC_SMEM = 220 * 1024;   // dynamic shared memory a launch may ask for

// Arrays of a level's region of shared memory, `pitch` elements each.
// The couplings downwards of line segments come from the cell below, and only
// FP64 levels store the inverse diagonal.
enum CcArray { A_DG, A_CE, A_CW, A_CN, A_CS, A_CT, A_B, A_X0, A_X1, A_LINES, A_CB = A_LINES, A_POINTS, A_DI = A_POINTS, A_NUM };

// Cells of the largest level that one block owns (FP64 issues a warp
// instruction in 16 cycles, so a whole block's step takes longer than the
// cluster's barrier).
template <typename T>
constexpr int SOLO = sizeof(T) == 8 ? 128 : 512;

template <typename T>
struct CcLevel {
    LevelView<T> v;
    const unsigned char *active;
    int f0, f1, f2;
    int sites;           // cells, or segments of the line smoother, i fastest
    int shift, chunk;    // a block owns chunk = 2^shift of them
    unsigned div0, div1; // ceil(2^32 / n0), ceil(2^32 / n1): exact quotients of the at most 2^16 sites
    int pitch;           // elements per array; the last one stays zero (ghost neighbours)
    unsigned off;        // byte offset of the region
};
template <typename T>
struct CcArgs {
    CcLevel<T> L[CC_LEVELS];
    int nl, solo;        // levels; the first that one block owns (nl - 1 at most)
    int degree, first_done, singular, ncoarse, ainv_smem;
    unsigned ainv_off;
    T first, c1[8], c2[8];
    const double *ainv;
    const int *map;
    const T *b, *x;      // level 0: right-hand side and (first_done) iterate
    T *out;
};

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned remote(unsigned local, int block)   // another block's shared address
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(block));
    return r;
}
__device__ __forceinline__ float ld_cluster(unsigned a, float)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double ld_cluster(unsigned a, double)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

// Site m of a level, 0-based.
struct Cell {
    int i, j, k;
};
template <typename T>
__device__ __forceinline__ Cell site(const CcLevel<T> &L, int m)
{
    // a divisor of 1 has no 32-bit ceil(2^32 / d)
    const int r = L.v.n0 > 1 ? (int)__umulhi((unsigned)m, L.div0) : m;
    const int k = L.v.n1 > 1 ? (int)__umulhi((unsigned)r, L.div1) : r;
    return Cell{m - r * L.v.n0, r - k * L.v.n1, k};
}

// One block's view of the cluster's shared memory.
template <typename T>
struct Ctx {
    unsigned char *smem;
    unsigned base;   // its shared-window address
    int rank;
    __device__ __forceinline__ T *arr(const CcLevel<T> &L, int a) const { return (T *)(smem + L.off) + (size_t)a * L.pitch; }
    // Address of element e of array `a` in block `owner`.
    __device__ __forceinline__ unsigned addr(const CcLevel<T> &L, int a, int e, int owner) const
    {
        const unsigned l = base + L.off + (unsigned)((a * L.pitch + e) * (int)sizeof(T));
        return owner == rank ? l : remote(l, owner);
    }
    __device__ __forceinline__ unsigned zero(const CcLevel<T> &L, int a) const { return addr(L, a, L.pitch - 1, rank); }
    // Site m, wherever it lives (row s of its segment on line levels).
    __device__ __forceinline__ unsigned at(const CcLevel<T> &L, int a, int m, int s = 0) const
    {
        return addr(L, a, (s << L.shift) + (m & (L.chunk - 1)), m >> L.shift);
    }
};

template <typename T>
__device__ __forceinline__ T load_dinv(const LevelView<T> &v, int c);
template <>
__device__ __forceinline__ float load_dinv<float>(const LevelView<float> &, int)
{
    return 0.f;   // formed from the diagonal
}
template <>
__device__ __forceinline__ double load_dinv<double>(const LevelView<double> &v, int c)
{
    return __ldg(v.dinv + c);
}
__device__ __forceinline__ float dinv_reg(float dg, float) { return jacobi_inv(dg); }
__device__ __forceinline__ double dinv_reg(double, double di) { return di; }
__device__ __forceinline__ bool active_reg(float dg, float) { return dg > 0.f; }
__device__ __forceinline__ bool active_reg(double, double di) { return __double_as_longlong(di) != 0; }

__device__ __forceinline__ void team_sync(bool solo)
{
    if (solo) __syncthreads();
    else cluster_sync();
}

// The operator of the block's own cells into shared memory, a batch of loads
// in flight per thread (and the right-hand side and iterate of the first level).
template <typename T, bool LINES>
__device__ void stage(const Ctx<T> &S, const CcLevel<T> &L, const T *__restrict__ b, const T *__restrict__ x)
{
    const LevelView<T> &v = L.v;
    constexpr int seg = LINES ? LINE_SEG : 1, U = LINES ? 4 : 1, NA = 9;
    for (int t0 = threadIdx.x; t0 < L.chunk * seg; t0 += CC_THREADS * U) {
        T w[U][NA];
        bool in[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int t = t0 + q * CC_THREADS, m = S.rank * L.chunk + (t & (L.chunk - 1));
            const Cell u = site(L, m);
            const int k = u.k * seg + (t >> L.shift);
            in[q] = t < L.chunk * seg && m < L.sites && k < v.n2;
            if (!in[q]) continue;
            const int c = (u.i + 1) + v.sy * (u.j + 1) + v.sz * (k + 1);
            w[q][0] = __ldg(v.diag + c);
            w[q][1] = __ldg(v.cE + c);
            w[q][2] = __ldg(v.cE + c - 1);
            w[q][3] = __ldg(v.cN + c);
            w[q][4] = __ldg(v.cN + c - v.sy);
            w[q][5] = __ldg(v.cT + c);
            if (!LINES) w[q][6] = __ldg(v.cT + c - v.sz);
            if (sizeof(T) == 8) w[q][7] = load_dinv(v, c);
            if (b) w[q][8] = b[c];
            if (!LINES && x) S.arr(L, A_X0)[t] = x[c];
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            if (!in[q]) continue;
            const int t = t0 + q * CC_THREADS;
            S.arr(L, A_DG)[t] = w[q][0];
            S.arr(L, A_CE)[t] = w[q][1];
            S.arr(L, A_CW)[t] = w[q][2];
            S.arr(L, A_CN)[t] = w[q][3];
            S.arr(L, A_CS)[t] = w[q][4];
            S.arr(L, A_CT)[t] = w[q][5];
            if (!LINES) S.arr(L, A_CB)[t] = w[q][6];
            if (sizeof(T) == 8) S.arr(L, A_DI)[t] = w[q][7];
            if (b) S.arr(L, A_B)[t] = w[q][8];
        }
    }
}

// ---- point levels ---------------------------------------------------------------

// A thread's cell of a level while it is smoothed.
template <typename T>
struct Point {
    bool in;
    int e;             // its place in the block's share
    Cell u;
    unsigned nb[6];    // neighbours' addresses in X0 (X1 is `flip` bytes on)
    T b, dg, di, x0, d, ce, cw, cn, cs, ct, cb;

    __device__ __forceinline__ void load(const Ctx<T> &S, const CcLevel<T> &L)
    {
        const LevelView<T> &v = L.v;
        e = threadIdx.x;
        const int m = S.rank * L.chunk + e;
        in = e < L.chunk && m < L.sites;
        if (!in) return;
        u = site(L, m);
        const int sy = v.n0, sz = v.n0 * v.n1;
        auto near = [&](bool inside, int mm) { return inside ? S.at(L, A_X0, mm) : S.zero(L, A_X0); };
        nb[0] = near(u.i + 1 < v.n0, m + 1);
        nb[1] = near(u.i > 0, m - 1);
        nb[2] = near(u.j + 1 < v.n1, m + sy);
        nb[3] = near(u.j > 0, m - sy);
        nb[4] = near(u.k + 1 < v.n2, m + sz);
        nb[5] = near(u.k > 0, m - sz);
        dg = S.arr(L, A_DG)[e];
        ce = S.arr(L, A_CE)[e]; cw = S.arr(L, A_CW)[e];
        cn = S.arr(L, A_CN)[e]; cs = S.arr(L, A_CS)[e];
        ct = S.arr(L, A_CT)[e]; cb = S.arr(L, A_CB)[e];
        di = dinv_reg(dg, sizeof(T) == 8 ? S.arr(L, A_DI)[e] : T(0));
        b = S.arr(L, A_B)[e];
    }
    __device__ __forceinline__ T residual(unsigned flip) const
    {
        const T z = T(0);
        const T xe = ld_cluster(nb[0] + flip, z), xw = ld_cluster(nb[1] + flip, z), xn = ld_cluster(nb[2] + flip, z),
                xs = ld_cluster(nb[3] + flip, z), xt = ld_cluster(nb[4] + flip, z), xb = ld_cluster(nb[5] + flip, z);
        return cheb_residual(b, dg, x0, xe, xw, xn, xs, xt, xb, ce, cw, cn, cs, ct, cb);
    }
    // one step from buffer p into the other; the first of the steps upwards
    // has no previous update: dn = (first dinv) r
    __device__ __forceinline__ void step(const Ctx<T> &S, const CcLevel<T> &L, int p, T c1, T c2, bool fresh)
    {
        if (!in) return;
        const T r = residual(p ? (unsigned)(L.pitch * (int)sizeof(T)) : 0u), w = fx_mul(c2, di);
        d = fresh ? fx_mul(w, r) : fx_fma(w, r, fx_mul(c1, d));   // as cheb_update
        x0 = fx_add(x0, d);
        S.arr(L, p ? A_X0 : A_X1)[e] = x0;
    }
};

// Steps before the restriction, and the residual of the result in the buffer
// that does not hold it.
template <typename T>
__device__ void down_points(const CcArgs<T> &a, const Ctx<T> &S, const CcLevel<T> &L, bool first_done, bool solo)
{
    Point<T> P;
    P.load(S, L);
    if (P.in) {
        T *x = S.arr(L, A_X0) + P.e;
        if (first_done) P.x0 = *x;
        else *x = P.x0 = fx_mul(fx_mul(a.first, P.di), P.b);
        P.d = P.x0;   // from a zero guess the first update is x itself
    }
    if (!first_done) team_sync(solo);
    int p = 0;
    for (int s = 1; s < a.degree; ++s, p ^= 1) {
        P.step(S, L, p, a.c1[s], a.c2[s], false);
        team_sync(solo);
    }
    if (P.in) S.arr(L, p ? A_X0 : A_X1)[P.e] = P.residual(p ? (unsigned)(L.pitch * (int)sizeof(T)) : 0u);
    team_sync(solo);
}

// The prolongation of level C's result and the steps after it.
template <typename T>
__device__ void up_points(const CcArgs<T> &a, const Ctx<T> &S, const CcLevel<T> &L, const CcLevel<T> &C, int ebuf,
                          T *out, bool solo)
{
    Point<T> P;
    P.load(S, L);
    int p = (a.degree - 1) & 1;
    if (P.in) {
        T *x = S.arr(L, p ? A_X1 : A_X0) + P.e;
        P.x0 = *x;
        if (active_reg(P.dg, P.di)) {
            const Cell u = P.u;
            const int pm = (u.i >> (L.f0 - 1)) + C.v.n0 * ((u.j >> (L.f1 - 1)) + C.v.n1 * (u.k >> (L.f2 - 1)));
            P.x0 = fx_add(P.x0, ld_cluster(S.at(C, ebuf, pm), T(0)));
        }
        *x = P.x0;
    }
    team_sync(solo);
    for (int s = 0; s < a.degree; ++s, p ^= 1) {
        P.step(S, L, p, a.c1[s], s ? a.c2[s] : a.first, s == 0);
        if (out && s == a.degree - 1) {
            if (P.in) out[(P.u.i + 1) + L.v.sy * (P.u.j + 1) + L.v.sz * (P.u.k + 1)] = P.x0;
        } else {
            team_sync(solo);
        }
    }
}

// ---- levels of line segments (k_cheb_line), one segment per thread; FP32 -----------

struct Line {
    bool in;
    int t, i, j, k0, nk;
    unsigned nb[4], lo, hi;   // first cell's neighbours in X0, the cells below and above the segment
    unsigned stride[4];       // bytes from one cell's neighbour to the next (0 on the walls' zero element)
    float cb0, inv[LINE_SEG], cp[LINE_SEG], dg[LINE_SEG], ct[LINE_SEG], xo[LINE_SEG], d[LINE_SEG];

    __device__ __forceinline__ void load(const Ctx<float> &S, const CcLevel<float> &L)
    {
        const LevelView<float> &v = L.v;
        t = threadIdx.x;
        const int m = S.rank * L.chunk + t;
        in = t < L.chunk && m < L.sites;
        if (!in) return;
        const Cell u = site(L, m);
        i = u.i;
        j = u.j;
        k0 = u.k * LINE_SEG;
        nk = min(LINE_SEG, v.n2 - k0);
        const unsigned st = (unsigned)(L.chunk * (int)sizeof(float));
        const int sy = v.n0, sz = v.n0 * v.n1;
        auto near = [&](int f, bool in, int mm, int s) {
            if (f < 4) stride[f < 4 ? f : 0] = in ? st : 0u;
            return in ? S.at(L, A_X0, mm, s) : S.zero(L, A_X0);
        };
        nb[0] = near(0, i + 1 < v.n0, m + 1, 0);
        nb[1] = near(1, i > 0, m - 1, 0);
        nb[2] = near(2, j + 1 < v.n1, m + sy, 0);
        nb[3] = near(3, j > 0, m - sy, 0);
        lo = near(4, k0 > 0, m - sz, LINE_SEG - 1);
        hi = near(5, k0 + nk < v.n2, m + sz, 0);
        cb0 = __ldg(v.cT + (i + 1) + v.sy * (j + 1) + v.sz * k0);
        float cpm = 0.f;
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) {
            const int e = min(s, nk - 1) * L.chunk + t;
            dg[s] = S.arr(L, A_DG)[e];
            ct[s] = S.arr(L, A_CT)[e];
        }
        // the elimination's pivots depend on the operator alone
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) {
            inv[s] = cp[s] = 0.f;
            const float w = s > 0 ? ct[s > 0 ? s - 1 : 0] : 0.f;
            if (s < nk && dg[s] > 0.f) {
                inv[s] = rcp_of<float>(fx_fma(w, cpm, dg[s]));
                cp[s] = fx_mul(s < nk - 1 ? -ct[s] : 0.f, inv[s]);
            }
            cpm = cp[s];
        }
    }
    __device__ __forceinline__ float side(int f, int s, unsigned flip) const   // column f's cell s
    {
        return ld_cluster(nb[f] + flip + s * stride[f], 0.f);
    }
    __device__ __forceinline__ void residuals(const Ctx<float> &S, const CcLevel<float> &L, unsigned flip,
                                              float (&r)[LINE_SEG]) const
    {
        const float xm0 = ld_cluster(lo + flip, 0.f), xp0 = ld_cluster(hi + flip, 0.f);
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) {
            const int q = min(s, nk - 1), e = q * L.chunk + t;
            const float xp = s == nk - 1 || s == LINE_SEG - 1 ? xp0 : xo[s + 1 < LINE_SEG ? s + 1 : s];
            const float xm = s ? xo[s - 1] : xm0, cb = s ? ct[s - 1] : cb0;
            r[s] = line_residual(S.arr(L, A_B)[e], dg[s], xo[s], side(0, q, flip),
                                 side(1, q, flip),
                                 side(2, q, flip),
                                 side(3, q, flip), xp, xm, S.arr(L, A_CE)[e],
                                 S.arr(L, A_CW)[e], S.arr(L, A_CN)[e], S.arr(L, A_CS)[e], ct[s], cb);
        }
    }
    // z = T^-1 r by substitution, then x += c1 d + c2 z
    __device__ __forceinline__ void finish(float (&r)[LINE_SEG], float c1, float c2, float *x, int chunk)
    {
        float ym = 0.f;
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) {
            const float w = s > 0 ? ct[s > 0 ? s - 1 : 0] : 0.f;
            r[s] = s < nk && dg[s] > 0.f ? fx_mul(fx_fma(w, ym, r[s]), inv[s]) : 0.f;
            ym = r[s];
        }
        float zn = 0.f;
#pragma unroll
        for (int s = LINE_SEG - 1; s >= 0; --s)
            if (s < nk) {
                const float z = fx_fma(-cp[s], zn, r[s]);
                zn = z;
                d[s] = line_dn(c1, d[s], c2, z);
                xo[s] = fx_add(xo[s], d[s]);
                x[s * chunk + t] = xo[s];
            }
    }
    __device__ __forceinline__ void step(const Ctx<float> &S, const CcLevel<float> &L, int p, float c1, float c2)
    {
        if (!in) return;
        float r[LINE_SEG];
        residuals(S, L, p ? (unsigned)(L.pitch * (int)sizeof(float)) : 0u, r);
        finish(r, c1, c2, S.arr(L, p ? A_X0 : A_X1), L.chunk);
    }
};

__device__ void down_lines(const CcArgs<float> &a, const Ctx<float> &S, const CcLevel<float> &L, bool solo)
{
    Line P;
    P.load(S, L);
    if (P.in) {   // from a zero guess: r = b, and the next step's previous update is x itself
        float r[LINE_SEG];
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) {
            r[s] = S.arr(L, A_B)[min(s, P.nk - 1) * L.chunk + P.t];
            P.xo[s] = P.d[s] = 0.f;
        }
        P.finish(r, 0.f, a.first, S.arr(L, A_X0), L.chunk);
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s) P.d[s] = P.xo[s];
    }
    team_sync(solo);
    int p = 0;
    for (int s = 1; s < a.degree; ++s, p ^= 1) {
        P.step(S, L, p, a.c1[s], a.c2[s]);
        team_sync(solo);
    }
    if (P.in) {   // k_restrict's residual, in the smoothers' point form
        const unsigned flip = p ? (unsigned)(L.pitch * (int)sizeof(float)) : 0u;
        float *r = S.arr(L, p ? A_X0 : A_X1);
        const float xm0 = ld_cluster(P.lo + flip, 0.f), xp0 = ld_cluster(P.hi + flip, 0.f);
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s)
            if (s < P.nk) {
                const int e = s * L.chunk + P.t;
                const float xp = s == P.nk - 1 || s == LINE_SEG - 1 ? xp0 : P.xo[s + 1 < LINE_SEG ? s + 1 : s];
                r[e] = cheb_residual(S.arr(L, A_B)[e], P.dg[s], P.xo[s], P.side(0, s, flip),
                                     P.side(1, s, flip),
                                     P.side(2, s, flip),
                                     P.side(3, s, flip), xp, s ? P.xo[s - 1] : xm0,
                                     S.arr(L, A_CE)[e], S.arr(L, A_CW)[e], S.arr(L, A_CN)[e], S.arr(L, A_CS)[e],
                                     P.ct[s], s ? P.ct[s - 1] : P.cb0);
            }
    }
    team_sync(solo);
}

__device__ void up_lines(const CcArgs<float> &a, const Ctx<float> &S, const CcLevel<float> &L, const CcLevel<float> &C,
                         bool coarsest, int ebuf, float *out, bool solo)
{
    Line P;
    P.load(S, L);
    const LevelView<float> &v = L.v;
    int p = (a.degree - 1) & 1;
    if (P.in) {
        float *x = S.arr(L, p ? A_X1 : A_X0);
#pragma unroll
        for (int s = 0; s < LINE_SEG; ++s)
            if (s < P.nk) {
                const int k = P.k0 + s, ci = P.i >> (L.f0 - 1), cj = P.j >> (L.f1 - 1), ck = k >> (L.f2 - 1);
                P.xo[s] = x[s * L.chunk + P.t];
                if (L.active[(P.i + 1) + v.sy * (P.j + 1) + v.sz * (k + 1)])
                    P.xo[s] = fx_add(P.xo[s],
                                     ld_cluster(coarsest ? S.at(C, ebuf, ci + C.v.n0 * (cj + C.v.n1 * ck))
                                                         : S.at(C, ebuf, ci + C.v.n0 * (cj + C.v.n1 * (ck / LINE_SEG)),
                                                                ck % LINE_SEG), 0.f));
                x[s * L.chunk + P.t] = P.xo[s];
                P.d[s] = P.xo[s];
            }
    }
    team_sync(solo);
    for (int s = 0; s < a.degree; ++s, p ^= 1) {
        P.step(S, L, p, s ? a.c1[s] : 0.f, s ? a.c2[s] : a.first);
        if (out && s == a.degree - 1) {
            if (P.in)
#pragma unroll
                for (int q = 0; q < LINE_SEG; ++q)
                    if (q < P.nk) out[(P.i + 1) + v.sy * (P.j + 1) + v.sz * (P.k0 + q + 1)] = P.xo[q];
        } else {
            team_sync(solo);
        }
    }
}

// ---- between levels -----------------------------------------------------------------

// The block's cells of level C: the children's residuals (in level F's buffer
// rbuf) summed in k_restrict's order -- j outer, k inner, from 0, for each of
// the two columns, then first + second -- and, for points, the first step.
template <typename T, bool LINES>
__device__ void restrict_level(const CcArgs<T> &a, const Ctx<T> &S, const CcLevel<T> &F, const CcLevel<T> &C, int rbuf,
                               bool to_coarsest, bool solo)
{
    const int seg = LINES && !to_coarsest ? LINE_SEG : 1;
    for (int t = threadIdx.x; t < C.chunk * seg; t += CC_THREADS) {
        const int l = t & (C.chunk - 1), q = t >> C.shift, m = S.rank * C.chunk + l;
        if (m >= C.sites) continue;
        const Cell w = site(C, m);
        const int i = w.i, j = w.j, k = w.k * seg + q;
        if (k >= C.v.n2) continue;
        T r[2][2][2];   // 0 outside the level
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int ii = i * F.f0 + (n & 1), jj = j * F.f1 + (n >> 1 & 1), kk = k * F.f2 + (n >> 2);
            T &v = r[n & 1][n >> 1 & 1][n >> 2];
            v = T(0);
            if ((n & 1) < F.f0 && (n >> 1 & 1) < F.f1 && (n >> 2) < F.f2 && ii < F.v.n0 && jj < F.v.n1 && kk < F.v.n2) {
                const int mm = ii + F.v.n0 * (jj + F.v.n1 * (LINES ? kk / LINE_SEG : kk));
                v = ld_cluster(S.at(F, rbuf, mm, LINES ? kk % LINE_SEG : 0), T(0));
            }
        }
        T col[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            col[u] = fx_add(fx_add(fx_add(fx_add(T(0), r[u][0][0]), r[u][0][1]), r[u][1][0]), r[u][1][1]);
        const T s = F.f0 == 2 ? fx_add(col[0], col[1]) : col[0];
        S.arr(C, A_B)[t] = s;
        if (!LINES && !to_coarsest)
            S.arr(C, A_X0)[l] = fx_mul(fx_mul(a.first, dinv_reg(S.arr(C, A_DG)[l],
                                                                sizeof(T) == 8 ? S.arr(C, A_DI)[l] : T(0))), s);
    }
    team_sync(solo);
}

// The coarsest level (k_coarse_solve), by the first block: the sums in that
// kernel's order, formed by the four warps that hold the unknowns alone, and
// one division.
template <typename T>
__device__ void coarsest(const CcArgs<T> &a, const Ctx<T> &S, const CcLevel<T> &L, const unsigned char *sact, double *sb,
                         double *red)
{
    __shared__ int cnt[4];
    const int t = threadIdx.x, n = a.ncoarse;
    const bool act = t < n && sact[t];
    double bv = t < n ? (double)S.arr(L, A_B)[t] : 0.0;
    if (a.singular) {
        if (t < 128) {
            double s = act ? bv : 0.0;
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            const unsigned w = __ballot_sync(0xffffffffu, act);
            if ((t & 31) == 0) { red[t >> 5] = s; cnt[t >> 5] = __popc(w); }
        }
        __syncthreads();
        if (t == 0) {
            const int c = cnt[0] + cnt[1] + cnt[2] + cnt[3];
            red[4] = c ? ((red[0] + red[2]) + (red[1] + red[3])) / (double)c : 0.0;
        }
        __syncthreads();
        if (act) bv -= red[4];
    }
    if (t < n) sb[t] = bv;
    __syncthreads();
    if (t < n) {
        double y = 0.0;
        if (a.ainv_smem) {   // stored by columns
            const double *A = (const double *)(S.smem + a.ainv_off);
#pragma unroll 8
            for (int s = 0; s < n; ++s) y += A[s * n + t] * sb[s];
        } else {
#pragma unroll 8
            for (int s = 0; s < n; ++s) y += a.ainv[(size_t)t * n + s] * sb[s];
        }
        S.arr(L, A_X0)[t] = act ? (T)y : T(0);
    }
    __syncthreads();
}

template <typename T, bool LINES>
__global__ void __launch_bounds__(CC_THREADS, 1) k_coarse_cycle(const __grid_constant__ CcArgs<T> a)
{
    after_previous();
    extern __shared__ __align__(16) unsigned char cc_smem[];
    __shared__ double sb[128], red[5];
    __shared__ unsigned char sact[128];
    Ctx<T> S;
    S.smem = cc_smem;
    S.base = (unsigned)__cvta_generic_to_shared(cc_smem);
    S.rank = blockIdx.x;   // the grid is one cluster
    const int last = a.nl - 1;
    for (int l = 0; l <= last; ++l) {
        const CcLevel<T> &L = a.L[l];
        if (threadIdx.x < 2) S.arr(L, threadIdx.x ? A_X1 : A_X0)[L.pitch - 1] = T(0);   // ghosts
        if (l == last) break;
        stage<T, LINES>(S, L, l ? nullptr : a.b, l || !a.first_done ? nullptr : a.x);
    }
    if (S.rank == 0 && threadIdx.x < a.ncoarse) sact[threadIdx.x] = a.L[last].active[a.map[threadIdx.x]];
    if (S.rank == 0 && a.ainv_smem) {
        const int n = a.ncoarse;
        double *A = (double *)(cc_smem + a.ainv_off);
        for (int e = threadIdx.x; e < n * n; e += CC_THREADS) A[(e % n) * n + e / n] = a.ainv[e];
    }
    cluster_sync();
    const int pre = (a.degree - 1) & 1, rbuf = pre ? A_X0 : A_X1;   // the iterate's parity, the residual's buffer
    auto down = [&](int l, bool solo) {
        const CcLevel<T> &L = a.L[l];
        if constexpr (LINES) {
            down_lines(a, S, L, solo);
        } else {
            const bool first = l > 0 || a.first_done;
            down_points<T>(a, S, L, first, solo);
        }
    };
    auto up = [&](int l, bool solo) {
        const CcLevel<T> &L = a.L[l], &C = a.L[l + 1];
        const int ebuf = l + 1 == last ? A_X0 : A_X1;   // a smoothed level ends after 2 degree - 1 exchanges
        T *out = l == 0 ? a.out : nullptr;
        if constexpr (LINES) {
            up_lines(a, S, L, C, l + 1 == last, ebuf, out, solo);
        } else {
            up_points<T>(a, S, L, C, ebuf, out, solo);
        }
    };
    for (int l = 0; l < a.solo; ++l) {
        down(l, false);
        restrict_level<T, LINES>(a, S, a.L[l], a.L[l + 1], rbuf, l + 1 == last, false);
    }
    if (S.rank == 0) {
        for (int l = a.solo; l < last; ++l) {
            down(l, true);
            restrict_level<T, LINES>(a, S, a.L[l], a.L[l + 1], rbuf, l + 1 == last, true);
        }
        coarsest<T>(a, S, a.L[last], sact, sb, red);
        for (int l = last - 1; l >= a.solo; --l) up(l, true);
    }
    if (a.solo > 0) {
        cluster_sync();
        for (int l = a.solo - 1; l >= 0; --l) up(l, false);
        cluster_sync();   // no block leaves while another reads its memory
    }
}

// Blocks of the cluster: 16 where the device can place one, else 8.
int cluster_blocks()
{
    static const int blocks = [] {
        for (int want : {CC_BLOCKS, 8}) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(want);
            cfg.blockDim = dim3(CC_THREADS);
            cfg.dynamicSmemBytes = CC_SMEM;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = want;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0, ok = 1;
            const void *fns[3] = {(const void *)k_coarse_cycle<float, false>, (const void *)k_coarse_cycle<float, true>,
                                  (const void *)k_coarse_cycle<double, false>};
            for (const void *f : fns)
                if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess || n < 1) ok = 0;
            cudaGetLastError();
            if (ok) return want;
        }
        return 0;
    }();
    return blocks;
}

// Fills the levels' shares and shared-memory layout; returns the bytes, 0 if
// a level does not fit a thread's cells.
template <typename T>
size_t plan(const MgLevel<T> *L, int nlev, bool lines, int blocks, CcArgs<T> *a)
{
    size_t off = 0;
    int solo = nlev - 1;
    for (int l = 0; l < nlev; ++l) {
        const MgLevel<T> &F = L[l];
        const bool seg = lines && l < nlev - 1;
        const long long sites = (long long)F.n0 * F.n1 * (seg ? (F.n2 + LINE_SEG - 1) / LINE_SEG : F.n2);
        const bool one = l == nlev - 1 || solo < l || sites <= SOLO<T>;
        if (one && l < solo) solo = l;
        int shift = 5;
        while ((1ll << shift) * (one ? 1 : blocks) < sites) ++shift;
        const long long chunk = 1ll << shift;
        if (l < nlev - 1 && chunk > CC_THREADS) return 0;
        const long long elems = chunk * (seg ? LINE_SEG : 1) + 4;
        if (a) {
            CcLevel<T> &C = a->L[l];
            C.v = F.view();
            C.active = F.active;
            C.f0 = F.f0; C.f1 = F.f1; C.f2 = F.f2;
            C.sites = (int)sites;
            C.shift = shift;
            C.chunk = (int)chunk;
            C.div0 = (unsigned)(((1ull << 32) + F.n0 - 1) / F.n0);
            C.div1 = (unsigned)(((1ull << 32) + F.n1 - 1) / F.n1);
            C.pitch = (int)elems;
            C.off = (unsigned)off;
        }
        off += (size_t)elems * (lines ? A_LINES : sizeof(T) == 8 ? A_NUM : A_POINTS) * sizeof(T);
        off = (off + 15) & ~(size_t)15;
    }
    const int nc = L[nlev - 1].n0 * L[nlev - 1].n1 * L[nlev - 1].n2;
    const size_t inv = (size_t)nc * nc * sizeof(double);
    const bool in = off + inv <= CC_SMEM;
    if (a) {
        a->nl = nlev;
        a->solo = solo;
        a->ainv_smem = in ? 1 : 0;
        a->ainv_off = (unsigned)off;
    }
    return in ? off + inv : off;
}

}  // namespace

cudaError_t coarse_cycle_attr()
{
    const void *fns[3] = {(const void *)k_coarse_cycle<float, false>, (const void *)k_coarse_cycle<float, true>,
                          (const void *)k_coarse_cycle<double, false>};
    for (const void *f : fns) {
        cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CC_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cluster_blocks();
    return cudaSuccess;
}

template <typename T>
int coarse_first_level(const MgLevel<T> *L, int nlev, bool lines)
{
    const int last = nlev - 1, blocks = cluster_blocks();
    if (blocks == 0 || (lines && sizeof(T) == 8)) return last;
    for (int l = nlev > CC_LEVELS ? nlev - CC_LEVELS : 0; l < last; ++l) {
        const size_t bytes = plan<T>(L + l, nlev - l, lines, blocks, nullptr);
        if (bytes > 0 && bytes <= CC_SMEM) return l;
    }
    return last;
}

template <typename T>
T *launch_coarse_cycle(const MgLevel<T> *L, int nlev, const ChebCoef &cc, const double *ainv, const int *map,
                       int ncoarse, bool singular, bool first_done, bool after_event, cudaStream_t st)
{
    CcArgs<T> a;
    cudaLaunchConfig_t cfg = {};
    cfg.dynamicSmemBytes = plan<T>(L, nlev, cc.lines != 0, cluster_blocks(), &a);
    a.degree = cc.degree;
    a.first_done = first_done ? 1 : 0;
    a.singular = singular ? 1 : 0;
    a.ncoarse = ncoarse;
    a.first = (T)cc.first;
    for (int s = 0; s < 8; ++s) { a.c1[s] = (T)cc.c1[s]; a.c2[s] = (T)cc.c2[s]; }
    a.ainv = ainv;
    a.map = map;
    a.b = L[0].b;
    a.x = L[0].x;
    a.out = L[0].xb;
    cfg.gridDim = dim3(cluster_blocks());
    cfg.blockDim = dim3(CC_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cfg.gridDim.x;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = after_event ? 1 : 2;   // (a kernel that also waits for an event is launched plainly)
    if constexpr (sizeof(T) == 4) {
        if (cc.lines) cudaLaunchKernelEx(&cfg, k_coarse_cycle<T, true>, a);
        else cudaLaunchKernelEx(&cfg, k_coarse_cycle<T, false>, a);
    } else {
        cudaLaunchKernelEx(&cfg, k_coarse_cycle<T, false>, a);
    }
    return a.out;
}

template int coarse_first_level<float>(const MgLevel<float> *, int, bool);
template int coarse_first_level<double>(const MgLevel<double> *, int, bool);
template float *launch_coarse_cycle<float>(const MgLevel<float> *, int, const ChebCoef &, const double *, const int *,
                                           int, bool, bool, bool, cudaStream_t);
template double *launch_coarse_cycle<double>(const MgLevel<double> *, int, const ChebCoef &, const double *, const int *,
                                             int, bool, bool, bool, cudaStream_t);
