// k_bicgstab.cu -- BiCGStab (van der Vorst, SIAM J. Sci. Stat. Comput. 13,
// 1992) on the Jacobi-scaled momentum systems of the predictor, templated on
// the vector type (FP64, or FP32 inside FP64 iterative refinement).
//
// One iteration is four passes:
//   U: p = r + beta (p - omega v) in place (the first step of a run takes
//      p = r)
//   P: v = A p; r0.v; then alpha
//   S: s = r - alpha v, formed at the 7 points; t = A s; t.s, t.t; omega
//   X: s again, x += alpha p + omega s, r = s - omega t; r0.r, r.r; beta,
//      and the stopping test
// s is never stored.  Each thread marches d.kz cells of one (i, j) column and
// keeps its share of the dot products in registers, so a block writes one
// partial sum per dot for 128 x kz cells; after each of P, S and X the
// partials are summed in a fixed order (so every run is bitwise
// reproducible) and the scalars updated, which stay in device memory: by the
// block that finishes last on grids up to LAST_MAX, else by a launch of one
// block.  (The launches were 4 to 5 us each, three per iteration: a predictor
// step at 67x53x75 in FP64 2570 us with them, 2280 without.)  The reduction after X sets `done` when
// ||r||^2 <= target or on a breakdown, and every kernel after that returns at
// once, so the host enqueues several iterations and reads the scalars once
// per batch.
#include "pred_kernels.h"
#include "scf_launch.cuh"

namespace pred {
namespace {

constexpr int NT = 128;

__device__ __forceinline__ bool finite_nonzero(double a) { return a != 0.0 && isfinite(a); }

// What a pass sums: r0.v; t.s and t.t; r0.r and r.r; ||r||^2, ||r_T||^2 and ||b||^2.
enum RedKind { BR_ALPHA, BR_OMEGA, BR_RHO, BR_RESID };
constexpr int red_sums(int kind) { return kind == BR_ALPHA ? 1 : kind == BR_RESID ? 3 : 2; }

struct Red {
    double *partials;   // 4 per block
    unsigned *finished; // blocks of the running pass that have; 0 between passes
    BcgScalars *sc;
    int want_bb;
};
// Blocks up to which the last one sums a pass.  The tail's registers (55 to 72
// against 32 to 40 without) leave room for nine FP32 blocks of P and S per SM
// and eight of X, and the FP32 passes live on warps in flight: beyond one such
// wave a launch costs less (a predictor step, mixed: 128x176x128, 1408 blocks,
// 7.36 ms with the sums in the last block of P and S and 6.31 without;
// 320x96x130, 2160 blocks, 11.9 and 11.0; X at 128x112x96, 1344 blocks, +9%).
// FP64 P and S are bound by their arithmetic and gain (320x96x130 24.4 ms with
// launches, 22.6 without; 128x176x128 13.4 and 13.7).
template <typename T>
constexpr int LAST_MAX = sizeof(T) == 4 ? 152 * 9 : 152 * 16;
constexpr int LAST_MAX_X = 152 * 8;

// The scalars from a pass's sums, by one warp (which divides in one go).
template <int KIND>
__device__ __forceinline__ void scalars(BcgScalars *sc, const double (&s)[red_sums(KIND)], int want_bb)
{
    const int lane = threadIdx.x & 31;   // blocks are 32 wide
    if constexpr (KIND == BR_ALPHA) {    // alpha = rho / (r0.v)
        if (lane) return;
        const double a = sc->rho / s[0];
        if (finite_nonzero(s[0]) && isfinite(a)) sc->alpha = a;
        else { sc->alpha = 0.0; sc->breakdown = 1; sc->done = 1; }
    } else if constexpr (KIND == BR_OMEGA) {
        // omega = (t.s) / (t.t); t.t = 0 means s = 0 (omega = 0 finishes)
        if (lane) return;
        const double w = s[1] > 0.0 ? s[0] / s[1] : 0.0;
        sc->omega = isfinite(w) ? w : 0.0;
    } else if constexpr (KIND == BR_RHO) {
        // beta = (rho_new / rho) (alpha / omega), rho = rho_new, rr, and the stopping test
        const double omega = sc->omega, num = lane == 1 ? sc->alpha : s[0], den = lane == 1 ? omega : sc->rho;
        const double quot = num / den, other = __shfl_sync(0xffffffffu, quot, 1);
        if (lane) return;
        sc->rr = s[1];
        sc->iters += 1;
        const double b = quot * other;
        if (finite_nonzero(s[0]) && omega != 0.0 && isfinite(b)) sc->beta = b;
        else { sc->beta = 0.0; sc->breakdown = 1; sc->done = 1; }
        sc->rho = s[0];
        if (!(s[1] > sc->target)) sc->done = 1;   // converged (or NaN: the host checks)
    } else {   // a fresh start (p = r on the next P)
        if (lane) return;
        sc->rr = s[0];
        sc->rho = s[1];
        if (want_bb) sc->bb = s[2];
        sc->alpha = 1.0;
        sc->omega = 1.0;
        sc->beta = 0.0;
        sc->breakdown = 0;
        sc->done = 0;
        sc->iters = 0;
    }
}

// The grid's sums from 1024 strided ones, a[q][j] of thread t < 128 being the
// one that starts at block t + 128 j: a tree over their index (512, 256, ...
// 1 apart), whose first three levels are the thread's own.  WIDE: the block has
// more threads, which hold none.
template <int KIND, bool WIDE>
__device__ __forceinline__ void red_tree(const Red &R, double (&a)[red_sums(KIND)][8], int t)
{
    constexpr int Q = red_sums(KIND);
    __shared__ double sh[Q][NT];
    if (!WIDE || t < NT) {
#pragma unroll
        for (int d = 4; d > 0; d >>= 1)
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int j = 0; j < d; ++j) a[q][j] += a[q][j + d];
#pragma unroll
        for (int q = 0; q < Q; ++q) sh[q][t] = a[q][0];
    }
    __syncthreads();
    if (t >= 32) return;
    double s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        s[q] = (sh[q][t] + sh[q][t + 64]) + (sh[q][t + 32] + sh[q][t + 96]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_down_sync(0xffffffffu, s[q], o);
    }
    scalars<KIND>(R.sc, s, R.want_bb);   // (s is the sums in lane 0)
}

// Sums the partials of nb blocks with 128 threads, eight strided sums each.
template <int KIND>
__device__ __forceinline__ void red_tail(const Red &R, int nb)
{
    constexpr int Q = red_sums(KIND);
    const int t = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    double a[Q][8];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j) a[q][j] = 0.0;
    for (int m = 0; m < nb; m += 8 * NT) {
        double p[Q][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = m + t + NT * j;
#pragma unroll
            for (int q = 0; q < Q; ++q) p[q][j] = e < nb ? __ldcg(R.partials + 4 * (long long)e + q) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (m + NT * j < nb)   // (an FP64 addition of nothing would still hold the pipe)
#pragma unroll
                for (int q = 0; q < Q; ++q) a[q][j] += p[q][j];
    }
    red_tree<KIND, false>(R, a, t);
}

// The end of a pass: the block's sums to its partials, and with LAST the
// grid's in the block that finishes last.  The products and the warp sums are
// formed in A (FP32 for the FP32 iteration: this GPU runs FP64 at 1/64 of the
// FP32 rate), the sums over the block's warps and over the blocks in FP64.
template <int KIND, bool LAST, typename A>
__device__ __forceinline__ void pass_end(A (&v)[red_sums(KIND)], const Red &R)
{
    constexpr int Q = red_sums(KIND);
    __shared__ double sh[NT / 32][4];
    __shared__ int last;
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int lane = tid & 31, warp = tid >> 5, nb = (int)(gridDim.x * gridDim.y * gridDim.z);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        A a = v[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sh[warp][q] = (double)a;
    }
    __syncthreads();
    if (tid == 0) {
        const long long blk = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            double a = 0.0;
            for (int w = 0; w < NT / 32; ++w) a += sh[w][q];
            R.partials[4 * blk + q] = a;
        }
        if (LAST) last = count_in(R.finished) == (unsigned)nb - 1u;
    }
    if constexpr (LAST) {
        __syncthreads();
        if (!last) return;
        if (tid == 0) *R.finished = 0;
        red_tail<KIND>(R, nb);
    }
}

// The sums of a grid of many blocks, in a launch of one block with a strided
// sum per thread: the additions of red_tail in its order, with the partials'
// loads spread over eight times the warps.  One / two sums back to back, by 128
// threads and by 1024: 3.0 / 5.1 us and 3.3 / 5.0 at 1344 blocks, 6.7 / 14.6 and
// 4.8 / 8.1 at 8192, where a predictor step (256^3 mixed) takes 38.9 ms, 43.5
// before.
template <int KIND>
__global__ void __launch_bounds__(8 * NT) k_red(Red R, int nb)
{
    after_previous();
    if (KIND != BR_RESID && R.sc->done) return;
    constexpr int Q = red_sums(KIND), U = 4;
    __shared__ double strided[Q][8 * NT];
    const int t = threadIdx.x;
    double v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = 0.0;
    for (int e = t; e < nb; e += U * 8 * NT) {
        double p[U][Q];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int b = e + u * 8 * NT;
                p[u][q] = b < nb ? __ldcg(R.partials + 4 * (long long)b + q) : 0.0;
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e - t + u * 8 * NT < nb)
#pragma unroll
                for (int q = 0; q < Q; ++q) v[q] += p[u][q];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) strided[q][t] = v[q];
    __syncthreads();
    double a[Q][8];
    if (t < NT)
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int j = 0; j < 8; ++j) a[q][j] = strided[q][t + NT * j];
    red_tree<KIND, true>(R, a, t);
}

template <int KIND>
void sum_blocks(const Red &R, int nb, cudaStream_t st)
{
    launch_after(k_red<KIND>, 1, 8 * NT, 0, st, R, nb);
}

template <typename T>
struct M6 {
    const T *w, *s, *b, *e, *n, *t;
};

// The column segment of a thread: cells (i, j, k0..k1); `in` is false for
// threads outside the grid (they still join the block reduction).
#define COLUMN                                                                \
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;                  \
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;                  \
    const int k0 = blockIdx.z * d.kz + 1;                                     \
    const int k1 = min(k0 + d.kz - 1, d.K);                                   \
    const bool in = i <= d.I && j <= d.J;                                     \
    const long long c0 = i + d.sy * j + d.sz * k0;

template <typename T, typename F>
__device__ __forceinline__ T apply_stencil(const M6<T> &m, const Dims &d, long long c, F X)
{
    return X(c) - (m.w[c] * X(c - 1) + m.s[c] * X(c - d.sy) + m.b[c] * X(c - d.sz) + m.e[c] * X(c + 1) +
                   m.n[c] * X(c + d.sy) + m.t[c] * X(c + d.sz));
}

template <typename T>
__global__ void __launch_bounds__(NT) k_bcg_u(Dims d, const T *__restrict__ r, T *__restrict__ p,
                                              const T *__restrict__ v, const BcgScalars *sc, int first)
{
    after_previous();
    if (sc->done) return;
    COLUMN
    if (!in) return;
    const T beta = (T)sc->beta, omega = (T)sc->omega;
    long long c = c0;
    if (first)
        for (int k = k0; k <= k1; ++k, c += d.sz) p[c] = r[c];
    else
        for (int k = k0; k <= k1; ++k, c += d.sz) p[c] = r[c] + beta * (p[c] - omega * v[c]);
}

template <typename T, bool LAST>
__global__ void __launch_bounds__(NT) k_bcg_p(Dims d, M6<T> m, const T *__restrict__ p, const T *__restrict__ r0,
                                              T *__restrict__ v, Red R)
{
    after_previous();
    if (R.sc->done) return;
    COLUMN
    T acc[1] = {T(0)};
    if (in) {
        auto P = [&](long long q) { return p[q]; };
        long long c = c0;
        for (int k = k0; k <= k1; ++k, c += d.sz) {
            const T y = apply_stencil(m, d, c, P);
            v[c] = y;
            acc[0] += r0[c] * y;
        }
    }
    pass_end<BR_ALPHA, LAST>(acc, R);
}

template <typename T, bool LAST>
__global__ void __launch_bounds__(NT) k_bcg_s(Dims d, M6<T> m, const T *__restrict__ r, const T *__restrict__ v,
                                              T *__restrict__ t, Red R)
{
    after_previous();
    if (R.sc->done) return;
    COLUMN
    T acc[2] = {T(0), T(0)};
    if (in) {
        const T alpha = (T)R.sc->alpha;
        auto S = [&](long long q) { return r[q] - alpha * v[q]; };
        long long c = c0;
        for (int k = k0; k <= k1; ++k, c += d.sz) {
            const T y = apply_stencil(m, d, c, S);
            t[c] = y;
            acc[0] += y * S(c);
            acc[1] += y * y;
        }
    }
    pass_end<BR_OMEGA, LAST>(acc, R);
}

template <typename T, bool LAST>
__global__ void __launch_bounds__(NT) k_bcg_x(Dims d, T *__restrict__ x, T *__restrict__ r,
                                              const T *__restrict__ r0, const T *__restrict__ p,
                                              const T *__restrict__ v, const T *__restrict__ t, Red R)
{
    after_previous();
    if (R.sc->done) return;
    COLUMN
    T acc[2] = {T(0), T(0)};
    if (in) {
        const T alpha = (T)R.sc->alpha, omega = (T)R.sc->omega;
        long long c = c0;
        for (int k = k0; k <= k1; ++k, c += d.sz) {
            const T s = r[c] - alpha * v[c];
            x[c] = x[c] + (alpha * p[c] + omega * s);
            const T rn = s - omega * t[c];
            r[c] = rn;
            acc[0] += r0[c] * rn;
            acc[1] += rn * rn;
        }
    }
    pass_end<BR_RHO, LAST>(acc, R);
}

// x += e (the FP32 correction of a refinement round), pointwise.
__global__ void __launch_bounds__(NT) k_xadd(Dims d, double *__restrict__ x, const float *__restrict__ e)
{
    after_previous();
    COLUMN
    if (!in) return;
    long long c = c0;
    for (int k = k0; k <= k1; ++k, c += d.sz) x[c] = x[c] + (double)e[c];
}

// r = b - A x in FP64 (x = NULL stands for x = 0: r = b without the stencil
// pass); ||r||^2, ||r_T||^2 of the stored vector (r32 when given, summed in
// FP32) and, with want_bb, ||b||^2.
template <bool LAST>
__global__ void __launch_bounds__(NT) k_resid64(Dims d, M6<double> m, const double *__restrict__ b,
                                                const double *__restrict__ x, double *__restrict__ r64,
                                                float *__restrict__ r32, Red R)
{
    after_previous();
    COLUMN
    double acc[3] = {0.0, 0.0, 0.0};
    if (in) {
        auto X = [&](long long q) { return x[q]; };
        float rt2 = 0.f;
        long long c = c0;
        for (int k = k0; k <= k1; ++k, c += d.sz) {
            const double r = x ? b[c] - apply_stencil(m, d, c, X) : b[c];
            if (r64) r64[c] = r;
            if (r32) {
                const float f = (float)r;
                r32[c] = f;
                rt2 += f * f;
            }
            acc[0] += r * r;
            if (R.want_bb) acc[2] += b[c] * b[c];
        }
        acc[1] = r32 ? (double)rt2 : acc[0];
    }
    pass_end<BR_RESID, LAST>(acc, R);
}

__global__ void k_set_target(BcgScalars *sc, double target)
{
    after_previous();
    sc->target = target;
    sc->done = 0;
    sc->iters = 0;
}

template <typename T>
M6<T> m6(const T *const m[6])
{
    return M6<T>{m[0], m[1], m[2], m[3], m[4], m[5]};
}

}  // namespace

int march_len(int I, int J, int K, long long blocks)
{
    const long long cols = (long long)((I + 31) / 32) * ((J + 3) / 4);
    int kz = 16;
    while (kz > 1 && cols * ((K + kz - 1) / kz) < blocks) kz /= 2;
    return kz;
}

dim3 solver_block() { return dim3(32, 4, 1); }
dim3 solver_grid(const Dims &d) { return dim3((d.I + 31) / 32, (d.J + 3) / 4, (d.K + d.kz - 1) / d.kz); }

template <typename T>
int bcg_iteration(const Dims &d, const T *const m[6], BcgVecs<T> &V, bool first, Reduce &R,
                   BcgScalars *sc, cudaStream_t st, cudaEvent_t *ev)
{
    const dim3 g = solver_grid(d), b = solver_block();
    const M6<T> M = m6(m);
    T *p = V.p, *v = V.v;
    if (ev) cudaEventRecord(ev[0], st);
    launch_after(k_bcg_u<T>, g, b, 0, st, d, V.r, p, v, sc, first ? 1 : 0);
    const Red red{R.partials, R.finished, sc, 0};
    const bool last = R.nblocks <= LAST_MAX<T>, last_x = R.nblocks <= LAST_MAX_X;
    auto *kp = last ? k_bcg_p<T, true> : k_bcg_p<T, false>;
    auto *ks = last ? k_bcg_s<T, true> : k_bcg_s<T, false>;
    auto *kx = last_x ? k_bcg_x<T, true> : k_bcg_x<T, false>;
    if (ev) cudaEventRecord(ev[1], st);
    launch_after(kp, g, b, 0, st, d, M, p, V.r0, v, red);
    if (ev) cudaEventRecord(ev[2], st);
    if (!last) sum_blocks<BR_ALPHA>(red, R.nblocks, st);
    if (ev) cudaEventRecord(ev[3], st);
    launch_after(ks, g, b, 0, st, d, M, V.r, v, V.t, red);
    if (ev) cudaEventRecord(ev[4], st);
    if (!last) sum_blocks<BR_OMEGA>(red, R.nblocks, st);
    if (ev) cudaEventRecord(ev[5], st);
    launch_after(kx, g, b, 0, st, d, V.x, V.r, V.r0, p, v, V.t, red);
    if (ev) cudaEventRecord(ev[6], st);
    if (!last_x) sum_blocks<BR_RHO>(red, R.nblocks, st);
    return 4 + (last ? 0 : 2) + (last_x ? 0 : 1);
}

int resid64(const Dims &d, const double *const m[6], const double *b, const double *x, double *r64, float *r32,
            bool want_bb, Reduce &R, BcgScalars *sc, cudaStream_t st)
{
    const Red red{R.partials, R.finished, sc, want_bb ? 1 : 0};
    const bool last = R.nblocks <= LAST_MAX_X;
    auto *k = last ? k_resid64<true> : k_resid64<false>;
    launch_after(k, solver_grid(d), solver_block(), 0, st, d, m6(m), b, x, r64, r32, red);
    if (!last) sum_blocks<BR_RESID>(red, R.nblocks, st);
    return last ? 1 : 2;
}

void set_target(BcgScalars *sc, double target, cudaStream_t st)
{
    k_set_target<<<1, 1, 0, st>>>(sc, target);
}

void xadd(const Dims &d, double *x, const float *e, cudaStream_t st)
{
    launch_after(k_xadd, solver_grid(d), solver_block(), 0, st, d, x, e);
}

template int bcg_iteration<double>(const Dims &, const double *const[6], BcgVecs<double> &, bool, Reduce &,
                                    BcgScalars *, cudaStream_t, cudaEvent_t *);
template int bcg_iteration<float>(const Dims &, const float *const[6], BcgVecs<float> &, bool, Reduce &,
                                   BcgScalars *, cudaStream_t, cudaEvent_t *);

}  // namespace pred
