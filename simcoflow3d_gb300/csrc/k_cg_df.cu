// k_cg_df.cu -- the CG of the mixed solver in double-float arithmetic.
//
// This GPU executes FP64 at 1/64 of its FP32 rate, and the FP64 CG kernels
// (operator apply, vector updates, dot products) were bound by that rate, not
// by memory.  In the mixed solver the CG vectors x, r, p, q therefore hold
// unevaluated sums hi + lo of two FP32 numbers (a "double-float", about 48
// significand bits), and the fine operator is split the same way (its FP32
// copy is the hi part; the assembly also writes the lo parts).  The
// arithmetic is the error-free transformations of Dekker and Knuth -- the
// two-sum and the FMA-based two-product -- with every FP32 operation an
// explicitly rounded intrinsic, so that no contraction changes them.  Each
// vector occupies the 8 bytes per cell of its FP64 counterpart (the FP64
// buffers are reused), so memory traffic is unchanged.  The dot products of
// the iteration -- (p, Ap), (r, z) and (r, r) -- are FP64: each cell's
// double-float values are widened to FP64 (the FP32 -> FP64 widening is done
// with integer operations, which are exact), multiplied with an FP64 FMA and
// accumulated in FP64 per thread, per block and across blocks.  That is two
// to four FP64 operations per cell and dot, which the memory-bound kernels
// hide.  The solution is converted back to FP64 at the end of a CG round and
// its residual is recomputed in FP64, so the stopping test on the true
// residual is unchanged.
#include "scf_df.cuh"
#include "scf_launch.cuh"
#include "scf_reduce.cuh"

namespace {

__device__ __forceinline__ float2 two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return make_float2(s, e);
}
// |a| >= |b|
__device__ __forceinline__ float2 quick_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    return make_float2(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ float2 dadd(float2 x, float2 y)
{
    const float2 s = two_sum(x.x, y.x);
    return quick_two_sum(s.x, __fadd_rn(s.y, __fadd_rn(x.y, y.y)));
}
__device__ __forceinline__ float2 dneg(float2 x) { return make_float2(-x.x, -x.y); }
__device__ __forceinline__ float2 dmul(float2 x, float2 y)
{
    const float p = __fmul_rn(x.x, y.x);
    float e = __fmaf_rn(x.x, y.x, -p);
    e = __fmaf_rn(x.x, y.y, e);
    e = __fmaf_rn(x.y, y.x, e);
    return quick_two_sum(p, e);
}
// the double-float form of d: hi = d rounded to FP32, lo = d - hi rounded
// to FP32, both on the integer pipe (scf_common.cuh)
__device__ __forceinline__ float2 dfrom(double d)
{
    const float hi = scf_to_f32(d);
    return make_float2(hi, scf_lo_part(d, hi));
}
__device__ __forceinline__ double dto(float2 x) { return (double)x.x + (double)x.y; }

__device__ __forceinline__ float2 ld(const float2 *__restrict__ v, int c) { return v[c]; }

#define DF_ZCHUNK(A)                                                   \
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;          \
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;          \
    const int k0 = blockIdx.z * kz + 1;                               \
    const int k1 = min(k0 + kz - 1, (A).hi.n2);                       \
    const bool in = i <= (A).hi.n0 && j <= (A).hi.n1;

// operator coefficient of cell c from its hi (FP32 copy) and lo parts
__device__ __forceinline__ float2 cf(const float *hi, const float *lo, int c) { return make_float2(hi[c], lo[c]); }

}  // namespace

// q = A p; alpha from (p, q) (FP64 products and sums), and in all-Neumann
// systems the mean of A p, which is zero in exact arithmetic (double-float
// per thread, FP64 across threads)
template <bool LAST>
__global__ void __launch_bounds__(128, 8) k_spmv_df(DfOp A, const float2 *__restrict__ p, float2 *__restrict__ q,
                                                 RedOut red, int kz)
{
    after_previous();
    DF_ZCHUNK(A);
    double v = 0.0;
    float2 sq = make_float2(0.f, 0.f);
    if (in) {
        const int sy = A.hi.sy, sz = A.hi.sz;
        int c = i + sy * j + sz * k0;
        float2 xm = ld(p, c - sz), x0 = ld(p, c), tb = cf(A.hi.cT, A.tlo, c - sz);
        // the six neighbour products are summed as a tree (short dependency
        // chains: the kernel is latency-bound, not memory-bound, otherwise);
        // one accumulator each keeps the kernel within 64 registers, eight
        // blocks per SM
        for (int k = k0; k <= k1; ++k, c += sz) {
            const float2 xp = ld(p, c + sz), tt = cf(A.hi.cT, A.tlo, c);
            const float2 sx = dadd(dmul(cf(A.hi.cE, A.elo, c), ld(p, c + 1)),
                                   dmul(cf(A.hi.cE, A.elo, c - 1), ld(p, c - 1)));
            const float2 syy = dadd(dmul(cf(A.hi.cN, A.nlo, c), ld(p, c + sy)),
                                    dmul(cf(A.hi.cN, A.nlo, c - sy), ld(p, c - sy)));
            const float2 sz2 = dadd(dmul(tt, xp), dmul(tb, xm));
            const float2 s = dadd(dadd(sx, syy), sz2);
            const float2 y = dadd(dmul(cf(A.hi.diag, A.dlo, c), x0), dneg(s));
            q[c] = y;
            v = fma(dwide(x0), dwide(y), v);
            sq = dadd(sq, y);
            xm = x0; x0 = xp; tb = tt;
        }
    }
    const double dv = block_sum(v);
    __syncthreads();
    double v2[2] = {dv, block_sum(dto(sq))};
    red_end<RK_ALPHA, LAST>(red, v2);
}

// (r, z) for beta: r double-float, z the FP32 preconditioned residual; FP64
// products and sums
template <bool LAST>
__global__ void __launch_bounds__(128) k_dot_rz_df(DfOp A, const float2 *__restrict__ r, const float *__restrict__ z,
                                                   RedOut red, int kz)
{
    after_previous();
    DF_ZCHUNK(A);
    double v = 0.0;
    if (in) {
        const int sy = A.hi.sy, sz = A.hi.sz;
        int c = i + sy * j + sz * k0;
        // four cells' loads in flight at a time
        for (int k = k0; k <= k1; k += 4) {
            float2 rr[4];
            float zz[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool on = k + u <= k1;
                rr[u] = on ? ld(r, c + u * sz) : make_float2(0.f, 0.f);
                zz[u] = on ? z[c + u * sz] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) v = fma(dwide(rr[u]), widen(zz[u]), v);
            c += 4 * sz;
        }
    }
    red_end<RK_BETA, LAST>(red, block_sum(v));
}

// x += alpha p, r -= alpha (q - mean q), (r, r) in FP64; also the FP32 copy
// of r (its hi part) for the V-cycle and, when x0 is given, the first
// point-Jacobi smoothing step from a zero guess, x0 = first D^-1 r.
template <bool LAST>
__global__ void __launch_bounds__(128) k_cg_update_df(DfOp A, float2 *__restrict__ x, float2 *__restrict__ r,
                                                      const float2 *__restrict__ p, const float2 *__restrict__ q,
                                                      float *__restrict__ rlow, float *__restrict__ x0, float first,
                                                      RedOut red, int kz)
{
    after_previous();
    DF_ZCHUNK(A);
    double v = 0.0;
    if (in) {
        const float2 al = dfrom(red.scal[S_ALPHA]), mal = dneg(al), qm = dfrom(red.scal[S_QMEAN]);
        const int sy = A.hi.sy, sz = A.hi.sz;
        int c = i + sy * j + sz * k0;
        for (int k = k0; k <= k1; ++k, c += sz) {
            x[c] = dadd(ld(x, c), dmul(al, ld(p, c)));
            const float dg = A.hi.diag[c];
            float2 qq = ld(q, c);
            if (dg > 0.f) qq = dadd(qq, dneg(qm));
            const float2 rn = dadd(ld(r, c), dmul(mal, qq));
            r[c] = rn;
            rlow[c] = rn.x;
            if (x0) x0[c] = first * jacobi_inv(dg) * rn.x;
            const double rd = dwide(rn);
            v = fma(rd, rd, v);
        }
    }
    red_end<RK_RR, LAST>(red, block_sum(v));
}

// p = z + beta p (p = z on the first call)
__global__ void __launch_bounds__(128) k_pupdate_df(DfOp A, const float *__restrict__ z, float2 *__restrict__ p,
                                                    const double *__restrict__ scal, int first, int kz)
{
    after_previous();
    DF_ZCHUNK(A);
    if (!in) return;
    const float2 be = dfrom(first ? 0.0 : scal[S_BETA]);
    const int sy = A.hi.sy, sz = A.hi.sz;
    int c = i + sy * j + sz * k0;
    for (int k = k0; k <= k1; ++k, c += sz) {
        const float2 zz = make_float2(z[c], 0.f);
        p[c] = first ? zz : dadd(zz, dmul(be, ld(p, c)));
    }
}

// element-wise conversions over the whole padded array (in place allowed)
__global__ void k_df_from_double(const double *src, float2 *dst, int n)
{
    after_previous();
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const double d = src[e];
        dst[e] = dfrom(d);
    }
}
// the residual at the start of a CG round: its double-float form in place
// and its FP32 copy (the hi part) for the V-cycle, in one pass
__global__ void k_df_round_start(double *r, float *rlow, int n)
{
    after_previous();
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const float2 v = dfrom(r[e]);
        ((float2 *)r)[e] = v;
        rlow[e] = v.x;
    }
}
__global__ void k_df_to_double(const float2 *src, double *dst, int n)
{
    after_previous();
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const float2 v = src[e];
        dst[e] = dwide(v);
    }
}

void df_spmv_dot(const DfOp &A, const float2 *p, float2 *q, Reducer &R, bool singular, cudaStream_t st,
                 int *launches, KTimer *kt)
{
    const March l = launch_march(A.hi.n0, A.hi.n1, A.hi.n2);
    const int id = kt_begin(kt, KC_SPMV, st);
    auto *k = red_last(nblocks(l)) ? k_spmv_df<true> : k_spmv_df<false>;
    launch_after(k, l.grid, l.block, 0, st, A, p, q, red_out(R, singular), l.kz);
    kt_end(kt, id, st);
    *launches += 1;
    red_finish<RK_ALPHA>(R, nblocks(l), singular, st, launches);
}

void df_dot_rz(const DfOp &A, const float2 *r, const float *z, Reducer &R, cudaStream_t st, int *launches)
{
    const March l = launch_march(A.hi.n0, A.hi.n1, A.hi.n2);
    auto *k = red_last(nblocks(l)) ? k_dot_rz_df<true> : k_dot_rz_df<false>;
    launch_after(k, l.grid, l.block, 0, st, A, r, z, red_out(R), l.kz);
    *launches += 1;
    red_finish<RK_BETA>(R, nblocks(l), false, st, launches);
}

void df_cg_update(const DfOp &A, float2 *x, float2 *r, const float2 *p, const float2 *q, float *rlow, float *x0,
                  double first, Reducer &R, cudaStream_t st, int *launches, KTimer *kt)
{
    const March l = launch_march(A.hi.n0, A.hi.n1, A.hi.n2);
    const int id = kt_begin(kt, KC_CGUPDATE, st);
    auto *k = red_last(nblocks(l)) ? k_cg_update_df<true> : k_cg_update_df<false>;
    launch_after(k, l.grid, l.block, 0, st, A, x, r, p, q, rlow, x0, (float)first, red_out(R), l.kz);
    kt_end(kt, id, st);
    *launches += 1;
    red_finish<RK_RR>(R, nblocks(l), false, st, launches);
}

void df_pupdate(const DfOp &A, const float *z, float2 *p, const double *scal, bool first, cudaStream_t st,
                int *launches)
{
    const March l = launch_march(A.hi.n0, A.hi.n1, A.hi.n2);
    launch_after(k_pupdate_df, l.grid, l.block, 0, st, A, z, p, scal, first ? 1 : 0, l.kz);
    *launches += 1;
}

void df_from_double(const double *src, float2 *dst, int n, cudaStream_t st, int *launches)
{
    launch_after(k_df_from_double, 152 * 8, 256, 0, st, src, dst, n);
    *launches += 1;
}

void df_round_start(double *r, float *rlow, int n, cudaStream_t st, int *launches)
{
    launch_after(k_df_round_start, 152 * 8, 256, 0, st, r, rlow, n);
    *launches += 1;
}

void df_to_double(const float2 *src, double *dst, int n, cudaStream_t st, int *launches)
{
    launch_after(k_df_to_double, 152 * 8, 256, 0, st, src, dst, n);
    *launches += 1;
}
