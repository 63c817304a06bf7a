// scf_cheb.cuh -- the arithmetic of the V-cycle's smoothers, shared by the
// kernels that run one level per launch (k_solver.cu) and the one that runs
// all small levels (k_coarse.cu), so that they agree bit for bit.
#pragma once
#include "scf_common.cuh"

// Jacobi scaling.  FP32 levels compute 1/diag on the fly with the hardware
// reciprocal (one instruction, and it saves one array per pass); FP64 levels
// read a stored inverse (FP64 division is slow on this GPU).  Inactive cells carry diag = -1 and
// get no update and no coarse correction.
template <typename T>
__device__ __forceinline__ T dinv_at(const LevelView<T> &L, int c);
template <>
__device__ __forceinline__ float dinv_at<float>(const LevelView<float> &L, int c)
{
    return jacobi_inv(L.diag[c]);
}
template <>
__device__ __forceinline__ double dinv_at<double>(const LevelView<double> &L, int c)
{
    return L.dinv[c];
}
template <typename T>
__device__ __forceinline__ bool active_at(const LevelView<T> &L, int c);
template <>
__device__ __forceinline__ bool active_at<float>(const LevelView<float> &L, int c)
{
    return L.diag[c] > 0.0f;
}
template <>
__device__ __forceinline__ bool active_at<double>(const LevelView<double> &L, int c)
{
    return __double_as_longlong(L.dinv[c]) != 0;
}

// Arithmetic of one Chebyshev update with every operation spelled out (no
// contraction left to the compiler), so that the one-step kernel and the
// fused two-step kernel give the same bits: the six neighbour products
// summed by FMA in the order E, W, N, S, T, B; A x = diag x - s;
// r = b - A x; the update dn = (c2 dinv) r + c1 dprev.
__device__ __forceinline__ float fx_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double fx_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fx_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fx_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fx_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double fx_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float fx_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double fx_add(double a, double b) { return __dadd_rn(a, b); }

// r = b - A x of one cell, the residual both the Chebyshev update and the
// restriction use, so a fused residual gives the bits of a separate one.
template <typename T>
__device__ __forceinline__ T cheb_residual(T b, T dg, T x0, T xe, T xw, T xn, T xs, T xt, T xb, T ce, T cw, T cn,
                                           T cs, T ct, T cb)
{
    T s = fx_mul(ce, xe);
    s = fx_fma(cw, xw, s);
    s = fx_fma(cn, xn, s);
    s = fx_fma(cs, xs, s);
    s = fx_fma(ct, xt, s);
    s = fx_fma(cb, xb, s);
    return fx_sub(b, fx_fma(dg, x0, -s));
}

template <typename T>
__device__ __forceinline__ T cheb_update(T b, T dg, T dinv, T x0, T xe, T xw, T xn, T xs, T xt, T xb, T ce, T cw,
                                         T cn, T cs, T ct, T cb, T dprev, T c1, T c2)
{
    const T r = cheb_residual(b, dg, x0, xe, xw, xn, xs, xt, xb, ce, cw, cn, cs, ct, cb);
    return fx_fma(fx_mul(c2, dinv), r, fx_mul(c1, dprev));
}

template <typename T>
__device__ __forceinline__ T rcp_of(T v);
template <>
__device__ __forceinline__ float rcp_of<float>(float v) { return __frcp_rn(v); }
template <>
__device__ __forceinline__ double rcp_of<double>(double v) { return 1.0 / v; }

// One cell's residual of a line segment (its k-neighbours come from registers)
// and the update that follows the segment's elimination, for the small levels.
// k_cheb_line has the same expressions in place: through these its loads were
// scheduled worse (256x128x128 projection 8.7 -> 9.4 ms).
template <typename T>
__device__ __forceinline__ T line_residual(T b, T dg, T x0, T xe, T xw, T xn, T xs, T xt, T xb, T ce, T cw, T cn,
                                           T cs, T ct, T cb)
{
    T sum = fx_fma(ce, xe, fx_mul(cw, xw));
    sum = fx_fma(cn, xn, sum);
    sum = fx_fma(cs, xs, sum);
    sum = fx_fma(ct, xt, sum);
    sum = fx_fma(cb, xb, sum);
    return fx_sub(b, fx_fma(dg, x0, -sum));
}
template <typename T>
__device__ __forceinline__ T line_dn(T c1, T dprev, T c2, T z)
{
    return fx_fma(c2, z, fx_mul(c1, dprev));
}
