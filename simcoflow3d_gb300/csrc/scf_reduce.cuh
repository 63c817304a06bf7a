// scf_reduce.cuh -- the end of a reducing kernel: block sums to grid sums and
// the CG scalars made of them.
//
// Up to one resident wave of blocks, the block that finishes last adds the
// partials itself, so a dot product costs no launch of its own; with more
// blocks a kernel of one block does.  (There the count of every block, which
// waits for the block's stores, and the registers of the tail cost more than
// the launch.  A projection, mixed, with the sums in launches / in the last
// block at any number of blocks: 256^3, 4096 blocks, 13.47 / 13.62 ms;
// 512x256x256 27.5 / 27.7; 147x93x121, 1920 blocks, 3.20 / 3.24; 192^3 and
// 256x128x128 the same.  At 40^3 it takes 1018 us with the launches and 1001
// without, at 64^3 in FP64, 1024 blocks, 2193 and 2175.)
// Either way the order of the additions is fixed: 1024 strided sums, then a
// tree over each 32 of them and one over the 32 results.  128 threads form it
// with the trees' upper levels as additions of registers -- 36 FP64 warp
// instructions, which the SM's FP64 pipe issues one in 16 cycles or more,
// where a shuffle tree in 1024 threads has 160.
#pragma once
#include "scf_kernels.h"
#include "scf_launch.cuh"

struct RedOut {
    double *part, *scal, *mail;
    unsigned *done;   // blocks that have finished; 0 between launches
    int n0;           // offset of the second sum's partials
    int singular;
};
inline RedOut red_out(const Reducer &R, bool singular = false)
{
    return RedOut{R.partials, R.scal, R.mail, R.done, R.max_blocks, singular ? 1 : 0};
}
inline bool red_last(unsigned blocks) { return blocks <= MARCH_WAVE; }

// What is summed: (p, q) and q; (r, z); (r, r); (b, b); b and the count of
// active cells; (r, r) and x.
enum RedKind { RK_ALPHA, RK_BETA, RK_RR, RK_BB, RK_COUNT, RK_RESIDUAL };
constexpr int red_sums(int kind) { return kind == RK_ALPHA || kind == RK_COUNT || kind == RK_RESIDUAL ? 2 : 1; }

// Sums of nb partials by 128 threads, and the scalars that follow from them.
template <int KIND>
__device__ __forceinline__ void red_tail(const RedOut &o, int nb)
{
    constexpr int Q = red_sums(KIND);
    __shared__ double wp[Q][32];
    double *scal = o.scal;
    const int t = thread_linear(), w = t >> 2, g = t & 3;
    double known = 0.0, count = 0.0;
    if (KIND == RK_ALPHA || KIND == RK_BETA) known = scal[S_RZ];
    if (KIND == RK_ALPHA || KIND == RK_RESIDUAL) count = scal[S_COUNT];
    // thread t holds strided sums g + 4 j, j < 8, of the tree w
    double a[Q][8];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j) a[q][j] = 0.0;
    for (int m = 0; m < nb; m += 1024) {
        double p[Q][8];
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int e = m + 32 * w + g + 4 * j;
                p[q][j] = e < nb ? __ldcg(o.part + q * o.n0 + e) : 0.0;
            }
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (m + 256 * (t >> 5) < nb)   // (an FP64 addition of nothing would still hold the pipe)
#pragma unroll
                for (int j = 0; j < 8; ++j) a[q][j] += p[q][j];
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int j = 0; j < d; ++j) a[q][j] += a[q][j + d];
    for (int d = 2; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < Q; ++q) a[q][0] += __shfl_down_sync(0xffffffffu, a[q][0], d);
    if (g == 0)
#pragma unroll
        for (int q = 0; q < Q; ++q) wp[q][w] = a[q][0];
    __syncthreads();
    if (t >= 32) return;
    double v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = wp[q][t];
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], d);
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = __shfl_sync(0xffffffffu, v[q], 0);
    if (t > 1) return;
    // to the waiting host without a copy of its own (scf_api.cu, await_mail)
    constexpr int mail = KIND == RK_RR ? MAIL_RR : KIND == RK_RESIDUAL ? MAIL_RESIDUAL : KIND == RK_BB ? MAIL_BB : -1;
    if (mail >= 0 && t == 0 && o.mail) *(volatile double *)(o.mail + (mail >= 0 ? mail : 0) * MAIL_STRIDE) = v[0];
    // lanes 0 and 1 form the two quotients of a kind in one division
    if constexpr (KIND == RK_ALPHA) {
        // alpha = (r, z) / (p, q); for an all-Neumann system also the mean of
        // q over the active cells.  That mean is zero in exact arithmetic (the
        // constant is the null vector of the symmetric operator); the CG update
        // subtracts the rounding that it carries, so that the recursive
        // residual stays in the range of the operator instead of collecting a
        // component that no iterate can remove.
        const double num = t ? v[1] : known, den = t ? count : v[0];
        const bool ok = t ? o.singular && count > 0.0 : v[0] != 0.0;
        scal[t ? S_QMEAN : S_ALPHA] = ok ? num / den : 0.0;
        if (t == 0) scal[S_PQ] = v[0];
    } else if constexpr (KIND == RK_BETA) {
        if (t == 0) {
            scal[S_BETA] = known != 0.0 ? v[0] / known : 0.0;
            scal[S_RZ] = v[0];
        }
    } else if constexpr (KIND == RK_RR) {
        if (t == 0) scal[S_RR] = v[0];
    } else if constexpr (KIND == RK_BB) {
        if (t == 0) scal[S_BB] = v[0];
    } else if constexpr (KIND == RK_COUNT) {
        if (t == 0) {
            scal[S_SUM] = v[0];
            scal[S_COUNT] = v[1];
            scal[S_MEAN] = v[1] > 0.0 ? v[0] / v[1] : 0.0;
        }
    } else if (t == 0) {
        scal[S_RR] = v[0];
        scal[S_MEANX] = count > 0.0 ? v[1] / count : 0.0;
    }
}

// The end of a block of 128 threads; v: its sums, in thread 0.  LAST: the last
// block finishes the reduction.
template <int KIND, bool LAST>
__device__ __forceinline__ void red_end(const RedOut &o, double (&v)[red_sums(KIND)])
{
    if (thread_linear() == 0)
#pragma unroll
        for (int q = 0; q < red_sums(KIND); ++q) o.part[q * o.n0 + block_linear()] = v[q];
    if constexpr (LAST) {
        __shared__ int last;
        const int nb = (int)(gridDim.x * gridDim.y * gridDim.z);
        if (thread_linear() == 0) last = count_in(o.done) == (unsigned)nb - 1u;
        __syncthreads();
        if (!last) return;
        if (thread_linear() == 0) *o.done = 0;
        red_tail<KIND>(o, nb);
    }
}
template <int KIND, bool LAST>
__device__ __forceinline__ void red_end(const RedOut &o, double s)
{
    double v[1] = {s};
    red_end<KIND, LAST>(o, v);
}

template <int KIND>
__global__ void __launch_bounds__(128) k_reduce(RedOut o, int nb)
{
    after_previous();
    red_tail<KIND>(o, nb);
}

// After a launch of `blocks` blocks: the sums, where its last block has not formed them.
template <int KIND>
void red_finish(const Reducer &R, unsigned blocks, bool singular, cudaStream_t st, int *launches)
{
    if (red_last(blocks)) return;
    launch_after(k_reduce<KIND>, 1, 128, 0, st, red_out(R, singular), (int)blocks);
    *launches += 1;
}
