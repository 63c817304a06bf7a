// transport_body.cuh -- the per-cell work of the CLSVOF interface transport
// (src/Clsvof.f90: Clsvof_Scheme 355-798 and the routines it calls), written
// once for the device kernels of k_transport.cu and, compiled by a host C++
// compiler, for the tests that run the same bodies on the CPU.
//
// Layout (column-major, i fastest): "ghosted" (0:I+1,0:J+1,0:K+1), "interior"
// (1:I,1:J,1:K), wall planes (J,K) for x, (I,K) for y, (I,J) for z.  Every
// body is a function of one cell (or one wall-plane point), so a kernel is a
// bounds test and one call.
//
// Expressions keep the reference's operation order; the kernels are built
// with -fmad=false and the host build with -ffp-contract=off, so sqrt,
// division and the products round alike on both, and x**3 and x**(1/3) are
// computed correctly rounded on both (cube, cbrt_like), so the device
// reproduces the host bit for bit.
#pragma once

#include <math.h>
#include <stddef.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define TR_HD __host__ __device__ inline
// Never inlined: FP64 work behind a branch that is rarely taken.  The compiler
// turns a short inline branch into unconditional arithmetic and a select, and
// FP64 operations are what bounds these kernels.
#define TR_RARE __host__ __device__ __noinline__
#else
#define TR_HD inline
#define TR_RARE inline
#endif

#if defined(TR_HOST_CHECK)
#include <stdio.h>
#include <stdlib.h>
#define TR_CHECK(cond, what)                                                            \
    do {                                                                                \
        if (!(cond)) {                                                                  \
            fprintf(stderr, "transport index out of range: %s (%s:%d)\n", what, __FILE__, __LINE__); \
            abort();                                                                    \
        }                                                                               \
    } while (0)
#else
#define TR_CHECK(cond, what) ((void)0)
#endif

namespace tr {

constexpr double VOFEPS = 1.0e-14;   // Clsvof.f90:32
constexpr double ETA = 0.075;        // Clsvof.f90:32
constexpr double TOLPAR = 1.0e-14;   // Clsvof.f90:35
constexpr int BAND = 4;              // band_width, Clsvof.f90:31
constexpr int NSUB = 6;              // nv, Clsvof.f90:31

struct Dims {
    int I, J, K;
    TR_HD size_t g(int i, int j, int k) const
    {
        TR_CHECK(i >= 0 && i <= I + 1 && j >= 0 && j <= J + 1 && k >= 0 && k <= K + 1, "ghosted");
        return (size_t)i + (size_t)(I + 2) * ((size_t)j + (size_t)(J + 2) * (size_t)k);
    }
    TR_HD size_t n(int i, int j, int k) const
    {
        TR_CHECK(i >= 1 && i <= I && j >= 1 && j <= J && k >= 1 && k <= K, "interior");
        return (size_t)(i - 1) + (size_t)I * ((size_t)(j - 1) + (size_t)J * (size_t)(k - 1));
    }
    TR_HD size_t interior() const { return (size_t)I * J * K; }
    TR_HD size_t ghosted() const { return (size_t)(I + 2) * (J + 2) * (K + 2); }
    TR_HD int len(int axis) const { return axis == 0 ? I : axis == 1 ? J : K; }
    // the first dimension of a wall plane normal to `axis`
    TR_HD int plane_lead(int axis) const { return axis == 0 ? J : I; }
    TR_HD size_t plane_size(int axis) const
    {
        return axis == 0 ? (size_t)J * K : axis == 1 ? (size_t)I * K : (size_t)I * J;
    }
};

struct Geo {   // cell centres and spacings, interior
    const double *x, *y, *z, *dx, *dy, *dz;
};

TR_HD double sgn(double a) { return copysign(1.0, a); }

TR_HD uint64_t bits_of(double v)
{
    union { double d; uint64_t u; } c;
    c.d = v;
    return c.u;
}
TR_HD double from_bits(uint64_t u)
{
    union { double d; uint64_t u; } c;
    c.u = u;
    return c.d;
}

// Tests and sign changes on the 32-bit halves: the compiler turns their
// 64-bit forms back into FP64 comparisons and negations.
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ uint32_t hi32(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t lo32(double v) { return (uint32_t)__double2loint(v); }
__device__ __forceinline__ double from_halves(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
#else
TR_HD uint32_t hi32(double v) { return (uint32_t)(bits_of(v) >> 32); }
TR_HD uint32_t lo32(double v) { return (uint32_t)bits_of(v); }
TR_HD double from_halves(uint32_t hi, uint32_t lo) { return from_bits(((uint64_t)hi << 32) | lo); }
#endif
TR_HD int exp_of(double v) { return (int)(hi32(v) >> 20) & 0x7ff; }
TR_HD bool is_zero(double v) { return ((hi32(v) & 0x7fffffffu) | lo32(v)) == 0; }
TR_HD bool is_plus_zero(double v) { return (hi32(v) | lo32(v)) == 0; }
TR_HD bool is_one(double v) { return ((hi32(v) ^ 0x3ff00000u) | lo32(v)) == 0; }
TR_HD bool is_finite(double v) { return exp_of(v) != 0x7ff; }
TR_HD bool same_bits(double a, double b) { return ((hi32(a) ^ hi32(b)) | (lo32(a) ^ lo32(b))) == 0; }
TR_HD double flip_if(double v, bool f) { return from_halves(hi32(v) ^ (f ? 0x80000000u : 0u), lo32(v)); }

// x / d.  When d is a normal power of two its reciprocal is exact and
// x * (1/d) is the same correctly rounded quotient, without an FP64
// division (about ten instructions on GB300's narrow FP64 pipes).  Uniform
// grids with power-of-two spacings, and divisions by 2 or by 1, take it.
TR_HD double divd(double x, double d)
{
    const uint64_t b = bits_of(d);
    const uint64_t e = (b >> 52) & 0x7FFull;
    if ((b & 0xFFFFFFFFFFFFFull) == 0 && e >= 1 && e <= 2045)
        return x * from_bits((b & 0x8000000000000000ull) | ((2046ull - e) << 52));
    return x / d;
}

// x**3.d0, rounded once: x*x split exactly by an FMA, times x split again,
// one rounding of the sum (Dekker's product; correct but for ties finer
// than 2^-100).  gfortran calls the math library's pow, which comes within a
// hair of this but in glibc lands on the wrong side of a near-tie for about
// 0.08% of arguments; the correctly rounded value is what every build of the
// reference approximates, and host and device compute it alike.
TR_HD double cube(double x)
{
    const double p = x * x;
    const double e1 = fma(x, x, -p);   // x*x = p + e1 exactly
    const double c = p * x;
    const double e2 = fma(p, x, -c);   // p*x = c + e2 exactly
    return c + fma(e1, x, e2);
}

// x**(1.d0/3.d0) = x**a, a = fl(1/3) = 1/3 - 2^-54/3, rounded once: the
// cube root c refined by one Newton step on the residual x - c^3 (exact
// products by FMA), times x**(-2^-54/3) = 1 - (2^-54/3) ln x (the next term
// is below 2^-90).  Whatever ulp the starting cbrt or log carry, the sum
// rounds to the same double on host and device.
TR_HD double cbrt_like(double x)
{
    if (!(x > 0.0) || isinf(x)) return pow(x, 1.0 / 3.0);
    const double c = cbrt(x);
    const double c2h = c * c, c2l = fma(c, c, -c2h);
    const double c3h = c2h * c, c3l = fma(c2h, c, -c3h) + c2l * c;
    const double d = ((x - c3h) - c3l) / (3.0 * c2h);
    const double g = -(0x1p-54 / 3.0) * log(x);
    return c + (d + c * g);
}

TR_HD double max3(double a, double b, double c)
{
    const double m = a > b ? a : b;
    return m > c ? m : c;
}
TR_HD double min3(double a, double b, double c)
{
    const double m = a < b ? a : b;
    return m < c ? m : c;
}

// Volume_Fraction_Calc (Clsvof.f90:1475-1550): the liquid volume of the
// box cut at distance s from its corner along the normal.
TR_HD double volume_fraction(double dx, double dy, double dz, double nxx, double nyy, double nzz, double s)
{
    const double nx1 = fabs(nxx), ny1 = fabs(nyy), nz1 = fabs(nzz);
    const double dx1 = max3(nx1 * dx, ny1 * dy, nz1 * dz);
    const double dz1 = min3(nx1 * dx, ny1 * dy, nz1 * dz);
    const double dy1 = nx1 * dx + ny1 * dy + nz1 * dz - dx1 - dz1;
    const double sm = dx1 + dy1 + dz1;
    const double sc = s < sm - s ? s : sm - s;
    if (s <= 0.0) return 0.0;
    if (s >= sm) return 1.0 * dx * dy * dz;
    double fc;
    if (sc <= dz1) {
        fc = cube(sc) / (6.0 * dx1 * dy1 * dz1);
    } else if (sc <= dy1) {
        fc = (sc * sc - dz1 * sc + dz1 * dz1 / 3.0) / (2.0 * dx1 * dy1);
    } else if (dx1 >= dy1 + dz1) {
        if (sc >= dy1 + dz1) {
            fc = (2.0 * sc - dy1 - dz1) / (2.0 * dx1);
        } else {
            fc = cube(sc) - cube(sc - dz1) - cube(sc - dy1);
            fc = fc / (6.0 * dx1 * dy1 * dz1);
        }
    } else {
        if (sc > dx1) fc = cube(sc) - cube(sc - dz1) - cube(sc - dy1) - cube(sc - dx1);
        else fc = cube(sc) - cube(sc - dz1) - cube(sc - dy1);
        fc = fc / (6.0 * dx1 * dy1 * dz1);
    }
    if (s <= 0.5 * sm) return fc * dx * dy * dz;
    return (1.0 - fc) * dx * dy * dz;
}

// Newton_Raphson (1462-1473), at most 200 steps (the reference has no cap).
TR_HD double newton(double a3, double a2, double a1, double a0, double sc)
{
    double delvar = 1.0e6;
    for (int it = 0; it < 200 && fabs(delvar) > 1.0e-6 * fabs(sc); ++it) {
        delvar = (a3 * cube(sc) + a2 * (sc * sc) + a1 * sc + a0) / (3.0 * a3 * (sc * sc) + 2.0 * a2 * sc + a1);
        sc = sc - delvar;
    }
    return sc;
}

// Cubic_Equation_Solve (1380-1398).
TR_HD double cubic(double fc, double dx1, double dy1, double dz1, double sc, bool case2)
{
    if (case2)
        return newton(1.0, -3.0 * (dy1 + dz1), 3.0 * (dy1 * dy1 + dz1 * dz1),
                      6.0 * fc * dx1 * dy1 * dz1 - (cube(dy1) + cube(dz1)), sc);
    return newton(2.0, -3.0 * (dx1 + dy1 + dz1), 3.0 * (dx1 * dx1 + dy1 * dy1 + dz1 * dz1),
                  6.0 * fc * dx1 * dy1 * dz1 - (cube(dx1) + cube(dy1) + cube(dz1)), sc);
}

// Find_Distance (1311-1378) with Final_Distance (1400-1408).
TR_HD double find_distance(double dx, double dy, double dz, double nxx, double nyy, double nzz, double f)
{
    const double nx1 = fabs(nxx), ny1 = fabs(nyy), nz1 = fabs(nzz);
    const double dx1 = max3(nx1 * dx, ny1 * dy, nz1 * dz);
    double dz1 = min3(nx1 * dx, ny1 * dy, nz1 * dz);
    if (fabs(dz1) < TOLPAR) dz1 = 0.0;
    double dy1 = nx1 * dx + ny1 * dy + nz1 * dz - dx1 - dz1;
    if (fabs(dy1) < TOLPAR) dy1 = 0.0;
    const double fc = f < 1.0 - f ? f : 1.0 - f;
    const double sm = dx1 + dy1 + dz1;
    const bool lower = f <= 0.5;
    double sc = 6.0 * fc * dx1 * dy1 * dz1;
    sc = sgn(sc) * cbrt_like(fabs(sc));
    if (sc < dz1) return lower ? sc : sm - sc;
    sc = 0.5 * dz1 + sqrt(2.0 * fc * dx1 * dy1 - dz1 * dz1 / 12.0);
    if (sc < dy1) return lower ? sc : sm - sc;
    sc = fc * dx1 + (dy1 + dz1) / 2.0;
    if (dx1 >= dy1 + dz1) {
        if (sc < dy1 + dz1) sc = cubic(fc, dx1, dy1, dz1, sc, true);
    } else if (sc >= dx1) {
        sc = cubic(fc, dx1, dy1, dz1, sc, false);
        if (sc < dx1) sc = cubic(fc, dx1, dy1, dz1, sc, true);
    } else {
        sc = cubic(fc, dx1, dy1, dz1, sc, true);
    }
    return lower ? sc : sm - sc;
}

// Isinterface (801-815): partly filled, or next to the opposite phase.  A
// bulk cell -- exactly +0 or 1 with its six neighbours holding the same
// bits -- fails every test below, so it is answered with integer compares
// and no FP64 work.
TR_HD bool is_interface(const Dims &D, const double *vfl, int i, int j, int k)
{
    const double v = vfl[D.g(i, j, k)];
    const uint64_t b = bits_of(v);
    if ((b == 0 || b == 0x3FF0000000000000ull) && bits_of(vfl[D.g(i - 1, j, k)]) == b &&
        bits_of(vfl[D.g(i + 1, j, k)]) == b && bits_of(vfl[D.g(i, j - 1, k)]) == b &&
        bits_of(vfl[D.g(i, j + 1, k)]) == b && bits_of(vfl[D.g(i, j, k - 1)]) == b &&
        bits_of(vfl[D.g(i, j, k + 1)]) == b)
        return false;
    const double jump = 1.0 - 2.1 * VOFEPS;
    bool flag = v > VOFEPS && v < 1.0 - VOFEPS;
    if (fabs(vfl[D.g(i - 1, j, k)] - v) >= jump) flag = true;
    if (fabs(vfl[D.g(i + 1, j, k)] - v) >= jump) flag = true;
    if (fabs(vfl[D.g(i, j - 1, k)] - v) >= jump) flag = true;
    if (fabs(vfl[D.g(i, j + 1, k)] - v) >= jump) flag = true;
    if (fabs(vfl[D.g(i, j, k - 1)] - v) >= jump) flag = true;
    if (fabs(vfl[D.g(i, j, k + 1)] - v) >= jump) flag = true;
    return flag;
}

// Normal_Vector_Irre's test | |grad phi| - 1 | < ETA on the sum of squares of a
// difference triple, without the square root: the rounded |1 - sqrt(s)| is below
// ETA exactly for OFF_LO <= s <= OFF_HI (sqrt and the subtraction are
// monotonic, so two bisections give the interval's ends).
constexpr double OFF_LO = 0x1.b6147ae147ae2p-1, OFF_HI = 0x1.27d70a3d70a3ep+0;
TR_HD double norm2(double vx, double vy, double vz) { return vx * vx + vy * vy + vz * vz; }
TR_HD int side_of(double sm, double sp)
{
    const bool m_in = sm >= OFF_LO && sm <= OFF_HI, m_off = sm < OFF_LO || sm > OFF_HI;   // neither for NaN
    const bool p_in = sp >= OFF_LO && sp <= OFF_HI, p_off = sp < OFF_LO || sp > OFF_HI;
    return (m_in && p_off) ? -1 : (m_off && p_in) ? 1 : 0;
}

// Neighbours of a cell by constant strides from its own index.
struct Around {
    const Dims &D;
    int i, j, k;
    size_t g0, n0, gy, gz, ny, nz;
    TR_HD Around(const Dims &D_, int i_, int j_, int k_)
        : D(D_), i(i_), j(j_), k(k_), g0(D_.g(i_, j_, k_)), n0(D_.n(i_, j_, k_)), gy((size_t)(D_.I + 2)),
          gz((size_t)(D_.I + 2) * (size_t)(D_.J + 2)), ny((size_t)D_.I), nz((size_t)D_.I * (size_t)D_.J)
    {
    }
    TR_HD size_t g(int a, int b, int c) const   // ghosted, offsets a, b, c
    {
        const size_t t = g0 + (ptrdiff_t)a + (ptrdiff_t)b * (ptrdiff_t)gy + (ptrdiff_t)c * (ptrdiff_t)gz;
        TR_CHECK(t == D.g(i + a, j + b, k + c), "ghosted neighbour");
        return t;
    }
    TR_HD size_t n(int a, int b, int c) const   // interior
    {
        const size_t t = n0 + (ptrdiff_t)a + (ptrdiff_t)b * (ptrdiff_t)ny + (ptrdiff_t)c * (ptrdiff_t)nz;
        TR_CHECK(t == D.n(i + a, j + b, k + c), "interior neighbour");
        return t;
    }
};

// Normal_Vector_Irre (2361-2456) for 1 < i < I, 1 < j < J, 1 < k < K: per
// axis a one-sided difference towards the side whose neighbour's gradient
// is within ETA of unit length when the other's is not, else the central
// one.  The neighbours' tangential differences are taken where the
// reference takes them (the x test's minus side at i-1 with the j and k
// differences, and so on).
TR_HD void normal_irre(const Dims &D, const Geo &G, const double *phi, int i, int j, int k, double &nxx,
                       double &nyy, double &nzz)
{
    const Around A(D, i, j, k);
    auto P = [&](int a, int b, int c) { return phi[A.g(a, b, c)]; };
    auto X = [&](int a, int b, int c) { return G.x[A.n(a, b, c)]; };
    auto Y = [&](int a, int b, int c) { return G.y[A.n(a, b, c)]; };
    auto Z = [&](int a, int b, int c) { return G.z[A.n(a, b, c)]; };
    auto Q = [](double num, double den) { return divd(num, den); };
    const double p0 = P(0, 0, 0), x0 = X(0, 0, 0), y0 = Y(0, 0, 0), z0 = Z(0, 0, 0);
    double vx, vy, vz, sm, sp;
    int o = i >= 3 ? -2 : -1;
    vx = Q(p0 - P(o, 0, 0), x0 - X(o, 0, 0));
    vy = Q(P(-1, 1, 0) - P(-1, -1, 0), Y(-1, 1, 0) - Y(-1, -1, 0));
    vz = Q(P(-1, 0, 1) - P(-1, 0, -1), Z(-1, 0, 1) - Z(-1, 0, -1));
    sm = norm2(vx, vy, vz);
    o = i <= D.I - 2 ? 2 : 1;
    vx = Q(P(o, 0, 0) - p0, X(o, 0, 0) - x0);
    vy = Q(P(1, 1, 0) - P(1, -1, 0), Y(1, 1, 0) - Y(1, -1, 0));
    vz = Q(P(1, 0, 1) - P(1, 0, -1), Z(1, 0, 1) - Z(1, 0, -1));
    sp = norm2(vx, vy, vz);
    const int sx = side_of(sm, sp);
    o = j >= 3 ? -2 : -1;
    vy = Q(p0 - P(0, o, 0), y0 - Y(0, o, 0));
    vx = Q(P(1, -1, 0) - P(-1, -1, 0), X(1, -1, 0) - X(-1, -1, 0));
    vz = Q(P(0, -1, 1) - P(0, -1, -1), Z(0, -1, 1) - Z(0, -1, -1));
    sm = norm2(vx, vy, vz);
    o = j <= D.J - 2 ? 2 : 1;
    vx = Q(P(1, 1, 0) - P(-1, 1, 0), X(1, 1, 0) - X(-1, 1, 0));
    vy = Q(P(0, o, 0) - p0, Y(0, o, 0) - y0);
    vz = Q(P(0, 1, 1) - P(0, 1, -1), Z(0, 1, 1) - Z(0, 1, -1));
    sp = norm2(vx, vy, vz);
    const int sy = side_of(sm, sp);
    vx = Q(P(1, 0, -1) - P(-1, 0, -1), X(1, 0, -1) - X(-1, 0, -1));
    vy = Q(P(0, 1, -1) - P(0, -1, -1), Y(0, 1, -1) - Y(0, -1, -1));
    o = k >= 3 ? -2 : -1;
    vz = Q(p0 - P(0, 0, o), z0 - Z(0, 0, o));
    sm = norm2(vx, vy, vz);
    vx = Q(P(1, 0, 1) - P(-1, 0, 1), X(1, 0, 1) - X(-1, 0, 1));
    vy = Q(P(0, 1, 1) - P(0, -1, 1), Y(0, 1, 1) - Y(0, -1, 1));
    o = k <= D.K - 2 ? 2 : 1;
    vz = Q(P(0, 0, o) - p0, Z(0, 0, o) - z0);
    sp = norm2(vx, vy, vz);
    const int sz = side_of(sm, sp);
    // towards the minus side (-1, 0), the plus side (0, 1) or central (-1, 1)
    int hi = sx == -1 ? 0 : 1, lo = sx == 1 ? 0 : -1;
    nxx = Q(P(hi, 0, 0) - P(lo, 0, 0), X(hi, 0, 0) - X(lo, 0, 0));
    hi = sy == -1 ? 0 : 1; lo = sy == 1 ? 0 : -1;
    nyy = Q(P(0, hi, 0) - P(0, lo, 0), Y(0, hi, 0) - Y(0, lo, 0));
    hi = sz == -1 ? 0 : 1; lo = sz == 1 ? 0 : -1;
    nzz = Q(P(0, 0, hi) - P(0, 0, lo), Z(0, 0, hi) - Z(0, 0, lo));
}

// Interface_Reconstruct (1216-1309) of one cell: the unit normal and the
// corner distance of an interface cell, zeros elsewhere.  Cells on the
// walls take clamped central differences; a vanishing gradient gives +z.
TR_HD void reconstruct(const Dims &D, const Geo &G, const double *vfl, const double *phi, int i, int j, int k,
                       double &n1, double &n2, double &n3, double &d1)
{
    n1 = n2 = n3 = d1 = 0.0;
    // a partly filled cell is an interface cell whatever its neighbours hold
    const double v = vfl[D.g(i, j, k)];
    if (!(v > VOFEPS && v < 1.0 - VOFEPS) && !is_interface(D, vfl, i, j, k)) return;
    if (i > 1 && i < D.I && j > 1 && j < D.J && k > 1 && k < D.K) {
        normal_irre(D, G, phi, i, j, k, n1, n2, n3);
    } else {
        const int ip = i + 1 < D.I ? i + 1 : D.I, im = i - 1 > 1 ? i - 1 : 1;
        const int jp = j + 1 < D.J ? j + 1 : D.J, jm = j - 1 > 1 ? j - 1 : 1;
        const int kp = k + 1 < D.K ? k + 1 : D.K, km = k - 1 > 1 ? k - 1 : 1;
        n1 = divd(phi[D.g(ip, j, k)] - phi[D.g(im, j, k)], G.x[D.n(ip, j, k)] - G.x[D.n(im, j, k)]);
        n2 = divd(phi[D.g(i, jp, k)] - phi[D.g(i, jm, k)], G.y[D.n(i, jp, k)] - G.y[D.n(i, jm, k)]);
        n3 = divd(phi[D.g(i, j, kp)] - phi[D.g(i, j, km)], G.z[D.n(i, j, kp)] - G.z[D.n(i, j, km)]);
    }
    const double temp = sqrt(n1 * n1 + n2 * n2 + n3 * n3);
    if (temp < 1.0e-14) {
        n1 = 0.0; n2 = 0.0; n3 = 1.0;
    } else {
        n1 = n1 / temp; n2 = n2 / temp; n3 = n3 / temp;
    }
    const size_t c = D.n(i, j, k);
    d1 = find_distance(G.dx[c], G.dy[c], G.dz[c], n1, n2, n3, v);
}

// East/West/North/South/Top/Bottom_Flux (1553-1688): the liquid crossing
// one face in one sub-step, per unit face area, from the upstream cell.
TR_HD double face_flux(int axis, int side, double nxx, double nyy, double nzz, double diss, double volf, double dx,
                       double dy, double dz, double wdt)
{
    if (wdt == 0.0) return 0.0;
    const double nn = axis == 0 ? nxx : axis == 1 ? nyy : nzz;
    const bool thin = side > 0 ? nn <= 0.0 : nn >= 0.0;
    double flux;
    if (axis == 0) {
        flux = thin ? volume_fraction(wdt, dy, dz, nxx, nyy, nzz, diss) / (wdt * dy * dz)
                    : (volf * dx * dy * dz - volume_fraction(dx - wdt, dy, dz, nxx, nyy, nzz, diss)) / (wdt * dy * dz);
    } else if (axis == 1) {
        flux = thin ? volume_fraction(dx, wdt, dz, nxx, nyy, nzz, diss) / (dx * wdt * dz)
                    : (volf * dx * dy * dz - volume_fraction(dx, dy - wdt, dz, nxx, nyy, nzz, diss)) / (dx * wdt * dz);
    } else {
        flux = thin ? volume_fraction(dx, dy, wdt, nxx, nyy, nzz, diss) / (dx * dy * wdt)
                    : (volf * dx * dy * dz - volume_fraction(dx, dy, dz - wdt, nxx, nyy, nzz, diss)) / (dx * dy * wdt);
    }
    return flux * wdt;
}

// The fields one directional sweep reads.
struct SweepIn {
    const double *vfl, *phi;                 // ghosted, before the sweep
    const double *nx, *ny, *nz, *dis;        // ghosted normals, interior corner distances
    const double *vel;                       // the axis' face velocity, ghosted
    const double *bc_vel, *bc_lvs;           // the low wall plane of the axis
    const double *vf_first, *ls_first;       // the sub-step's first sweep result (later sweeps)
    double dtv;
    int axis, stage;                         // stage 0, 1, 2 within the sub-step
};

// A cell of the line along `axis` through (a, b): x lines are (j, k),
// y lines (i, k), z lines (i, j).
TR_HD size_t line_g(const Dims &D, int axis, int m, int a, int b)
{
    return axis == 0 ? D.g(m, a, b) : axis == 1 ? D.g(a, m, b) : D.g(a, b, m);
}
TR_HD size_t line_n(const Dims &D, int axis, int m, int a, int b)
{
    return axis == 0 ? D.n(m, a, b) : axis == 1 ? D.n(a, m, b) : D.n(a, b, m);
}

// Whether cell q is the upstream one of the face between cells q and q+1
// of a line: z tests w >= 0 where x and y test > 0 (X_Sweep 835-860 and its
// y, z forms).
TR_HD bool face_down(int axis, double w) { return axis == 2 ? w >= 0.0 : w > 0.0; }

// A partly filled cell, whose outflow is a geometric cut; a full or empty
// upstream cell sends vfl*u*dt.
TR_RARE bool partial_rare(double v) { return !(v >= 1.0 - VOFEPS || v <= VOFEPS); }
TR_HD bool partial_cell(double v)
{
    if (is_plus_zero(v) || is_one(v)) return false;   // without FP64 compares
    return partial_rare(v);
}

// The VOF flux through the face between cells q and q+1 of a line.
TR_HD double vof_face(const Dims &D, const Geo &G, const SweepIn &S, int q, int a, int b)
{
    const double w = S.vel[line_g(D, S.axis, q, a, b)];
    const bool down = face_down(S.axis, w);
    const int up = down ? q : q + 1;
    const size_t gu = line_g(D, S.axis, up, a, b), nu = line_n(D, S.axis, up, a, b);
    const double v = S.vfl[gu];
    if (!partial_cell(v)) return v * w * S.dtv;
    if (down) return face_flux(S.axis, +1, S.nx[gu], S.ny[gu], S.nz[gu], S.dis[gu], v, G.dx[nu], G.dy[nu], G.dz[nu],
                               w * S.dtv);
    return -face_flux(S.axis, -1, S.nx[gu], S.ny[gu], S.nz[gu], S.dis[gu], v, G.dx[nu], G.dy[nu], G.dz[nu], -w * S.dtv);
}

// The geometric fluxes a partial cell (i, j, k) with plane n.x = s sends
// through its faces along the axis: fh where it is upstream of its high
// face, fl where it is upstream of its low face (0 otherwise; nothing reads
// those).
TR_HD void partial_fluxes(const Dims &D, const Geo &G, const SweepIn &S, int i, int j, int k, double n1, double n2,
                          double n3, double s, double &fl, double &fh)
{
    const int ax = S.axis, n = D.len(ax), m = ax == 0 ? i : ax == 1 ? j : k;
    const size_t g = D.g(i, j, k), c = D.n(i, j, k);
    const double v = S.vfl[g], dx = G.dx[c], dy = G.dy[c], dz = G.dz[c];
    fl = fh = 0.0;
    if (m <= n - 1) {
        const double w = S.vel[g];
        if (face_down(ax, w)) fh = face_flux(ax, +1, n1, n2, n3, s, v, dx, dy, dz, w * S.dtv);
    }
    if (m >= 2) {
        const double w = S.vel[ax == 0 ? D.g(i - 1, j, k) : ax == 1 ? D.g(i, j - 1, k) : D.g(i, j, k - 1)];
        if (!face_down(ax, w)) fl = -face_flux(ax, -1, n1, n2, n3, s, v, dx, dy, dz, -w * S.dtv);
    }
}

// The level-set flux u*phi_face*dt through the face on the high side of
// cell q, phi_face extrapolated half a step upstream; q = 1 and q = n take
// the reference's boundary forms (x's backward difference /2*dx(2), z's
// plus sign, z's last face scaled by dy).
TR_HD double ls_face(const Dims &D, const Geo &G, const SweepIn &S, const double *d, const double *c, int q, int a,
                     int b)
{
    const int n = D.len(S.axis), ax = S.axis;
    auto PH = [&](int m) { return S.phi[line_g(D, ax, m, a, b)]; };
    auto DD = [&](int m) { return d[line_n(D, ax, m, a, b)]; };
    auto CC = [&](int m) { return c[line_n(D, ax, m, a, b)]; };
    const double w = S.vel[line_g(D, ax, q, a, b)], dtv = S.dtv;
    double ls;
    if (q == 1) {
        if (w >= 0.0) {
            const double den = ax == 0 ? DD(1) : CC(2) - CC(1);
            ls = PH(1) + divd(divd(DD(1), 2.0) * (1.0 - divd(w * dtv, DD(1))) * (PH(2) - PH(1)), den);
        } else if (ax == 0) {
            ls = PH(2) - divd(divd(DD(2), 2.0) * (1.0 + divd(w * dtv, DD(2))) * (PH(3) - PH(1)), 2.0) * DD(2);
        } else if (ax == 1) {
            ls = PH(2) - divd(divd(DD(2), 2.0) * (1.0 + divd(w * dtv, DD(2))) * (PH(3) - PH(1)), CC(3) - CC(1));
        } else {
            ls = PH(2) + divd(divd(DD(2), 2.0) * (1.0 + divd(w * dtv, DD(2))) * (PH(3) - PH(1)), CC(3) - CC(1));
        }
        return ls * w * dtv;
    }
    if (q == n) {
        if (w > 0.0) {
            ls = PH(n) + divd(divd(DD(n), 2.0) * (1.0 - divd(w * dtv, DD(n))) * (PH(n) - PH(n - 1)), CC(n) - CC(n - 1));
        } else {
            const double scale = ax == 2 ? G.dy[line_n(D, ax, n - 1, a, b)] : DD(n - 1);
            ls = PH(n) - divd(divd(DD(n - 1), 2.0) * (1.0 + divd(w * dtv, scale)) * (PH(n) - PH(n - 1)),
                              CC(n) - CC(n - 1));
        }
        return ls * w * dtv;
    }
    const double dm = DD(q), half = divd(dm, 2.0), step = divd(w * dtv, dm);
    if (w >= 0.0) ls = PH(q) + divd(half * (1.0 - step) * (PH(q + 1) - PH(q - 1)), 2.0 * dm);
    else if (q <= n - 2) ls = PH(q + 1) - divd(half * (1.0 + step) * (PH(q + 2) - PH(q)), 2.0 * dm);
    else ls = PH(q + 1) - divd(half * (1.0 + step) * (PH(q + 1) - PH(q)), dm);
    return w * ls * dtv;
}

// One cell of one sweep from the fluxes through its low and high faces (VOF
// vl, vh; level set ll, lh), added in the order the reference's face loops
// add them to this cell, then the sub-step's divergence term -- the first
// sweep divides by 1 - dtv/d (u_m - u_{m-1}), the later two add dtv/d
// times the first sweep's result times that difference -- and the clip of
// the VOF to 0 and 1 within 1e-14 (Clsvof_Scheme 486-780).  Needs n >= 3;
// vl and ll are not read at m = 1, vh not at m = n.
TR_HD void sweep_update(const Dims &D, const Geo &G, const SweepIn &S, int i, int j, int k, double vl, double vh,
                        double ll, double lh, double &vf_out, double &ls_out)
{
    const int ax = S.axis, n = D.len(ax);
    const int m = ax == 0 ? i : ax == 1 ? j : k;
    const int a = ax == 0 ? j : i, b = ax == 2 ? j : k;
    const double *d = ax == 0 ? G.dx : ax == 1 ? G.dy : G.dz;
    const size_t g = D.g(i, j, k), nc = D.n(i, j, k);
    const double dm = d[nc];
    const size_t gm = ax == 0 ? D.g(i - 1, j, k) : ax == 1 ? D.g(i, j - 1, k) : D.g(i, j, k - 1);
    const double ug = S.vel[g], um = S.vel[gm];
    // VOF (X_Sweep 835-875)
    const double v0 = S.vfl[g];
    double tv = v0;
    if (m >= 2) tv = tv + divd(vl, dm);
    if (m <= n - 1) tv = tv - divd(vh, dm);
    if (m == 1) {
        const double flux = v0 * um * S.dtv;
        tv = tv + divd(flux, dm);
    }
    if (m == n) {
        const double flux = v0 * ug * S.dtv;
        tv = tv - divd(flux, dm);
    }
    // level set (X_Sweep 877-947)
    double tl = S.phi[g];
    if (m >= 3) tl = tl + divd(ll, dm);
    tl = tl - divd(lh, dm);
    if (m == 1) {
        const size_t bw = (size_t)(a - 1) + (size_t)D.plane_lead(ax) * (size_t)(b - 1);
        TR_CHECK(bw < D.plane_size(ax), "wall plane");
        const double flux = S.bc_vel[bw] * S.bc_lvs[bw] * S.dtv;
        tl = tl + divd(flux, dm);
    }
    if (m == 2) tl = tl + divd(ll, dm);
    // the divergence term and the clip
    const double du = ug - um;
    const double rate = divd(S.dtv, dm);
    if (S.stage == 0) {
        const double den = 1.0 - rate * du;
        tv = divd(tv, den);
        tl = divd(tl, den);
    } else {
        tv = tv + rate * S.vf_first[g] * du;
        tl = tl + rate * S.ls_first[g] * du;
    }
    if (tv <= VOFEPS) tv = 0.0;
    if (tv >= 1.0 - VOFEPS) tv = 1.0;
    vf_out = tv;
    ls_out = tl;
}

// One cell of one sweep, gathered: both faces computed from the fields.
TR_HD void sweep_cell(const Dims &D, const Geo &G, const SweepIn &S, int i, int j, int k, double &vf_out,
                      double &ls_out)
{
    const int ax = S.axis, n = D.len(ax);
    const int m = ax == 0 ? i : ax == 1 ? j : k;
    const int a = ax == 0 ? j : i, b = ax == 2 ? j : k;
    const double *d = ax == 0 ? G.dx : ax == 1 ? G.dy : G.dz;
    const double *c = ax == 0 ? G.x : ax == 1 ? G.y : G.z;
    const double vl = m >= 2 ? vof_face(D, G, S, m - 1, a, b) : 0.0;
    const double vh = m <= n - 1 ? vof_face(D, G, S, m, a, b) : 0.0;
    const double ll = m >= 2 ? ls_face(D, G, S, d, c, m - 1, a, b) : 0.0;
    const double lh = ls_face(D, G, S, d, c, m, a, b);
    sweep_update(D, G, S, i, j, k, vl, vh, ll, lh, vf_out, ls_out);
}

// ---- the sweeps with shared work -------------------------------------------
//
// The same update as sweep_cell, bit for bit, with fewer FP64 operations (FP64
// issues at 2 lanes per clock per SM on GB300 and bounds the sweeps): every
// face once, quotients by a spacing through its reciprocal and kept while the
// spacing's bits repeat along the line, nothing computed for empty cells, and
// comparisons, halvings and sign tests on the integer pipe.


// x / 2, by the exponent where that stays normal.
TR_RARE double half_rare(double x) { return x / 2.0; }
TR_HD double half_of(double x)
{
    const int e = exp_of(x);
    if (e > 1 && e < 0x7ff) return from_halves(hi32(x) - 0x100000u, lo32(x));
    return half_rare(x);
}

// A cell's spacing along the line with what is formed from it.
struct LineStep {
    double d, r, r2; // r = 1/d, rounded; for a power of two exact, and r2 = 1/(2d)
    double half;     // d/2
    double rate;     // dtv / d
    bool pow2;
};

// x / d, correctly rounded, r = 1/d rounded: Markstein's division (IBM J. Res.
// Dev. 34, 1990).  One remainder step makes the quotient faithful and a second
// one, whose remainder is exact, rounds it correctly; five operations against
// about nine.  Outside the exponents where the remainders are exact, and for
// zeros, the division.
TR_RARE double div_rare(double x, double d, double r)
{
    const int e = exp_of(x), ed = exp_of(d);
    if (ed > 723 && ed < 1323 && e > 423 && e < 1623) {
        double q = x * r;
        q = fma(fma(-d, q, x), r, q);
        return fma(fma(-d, q, x), r, q);
    }
    return x / d;
}
// x / (2d) is half of x / d while both stay normal.
TR_RARE double div2_rare(double x, double d, double r)
{
    const double q = div_rare(x, d, r);
    const int e = exp_of(q), ed = exp_of(d);
    if (ed > 723 && ed < 1323 && e > 1 && e < 0x7ff) return half_of(q);
    return divd(x, 2.0 * d);
}
TR_HD double line_div(const LineStep &s, double x) { return s.pow2 ? x * s.r : div_rare(x, s.d, s.r); }
TR_HD double line_div2(const LineStep &s, double x) { return s.pow2 ? x * s.r2 : div2_rare(x, s.d, s.r); }

TR_RARE double recip_rare(double d) { return 1.0 / d; }
TR_HD LineStep line_step(double d, double dtv)
{
    LineStep s;
    s.d = d;
    const uint32_t h = hi32(d), e = (h >> 20) & 0x7ffu, sign = h & 0x80000000u;
    s.pow2 = ((h & 0xfffffu) | lo32(d)) == 0 && e >= 2 && e <= 2044;
    s.r2 = from_halves(sign | ((2045u - e) << 20), 0u);
    if (s.pow2) s.r = from_halves(sign | ((2046u - e) << 20), 0u);
    else s.r = recip_rare(d);
    s.half = half_of(d);
    s.rate = line_div(s, dtv);
    return s;
}

// The face between cells q and q + 1 of a line: its VOF and level-set fluxes,
// their quotients by cell q's spacing, and that spacing.
struct LineFace {
    double v, l, qv, ql, d;
};

// The VOF flux of a face whose upstream cell is neither empty nor full.
TR_RARE double vof_flux_rare(double v, double w, double dtv, const double *cut)
{
    return partial_cell(v) ? *cut : v * w * dtv;
}
TR_RARE double ls_face_rare(const Dims &D, const Geo &G, const SweepIn &S, const double *d, const double *c, int q,
                            int a, int b)
{
    return ls_face(D, G, S, d, c, q, a, b);
}

// s: cell q's spacing.  flo, fhi: the fluxes k_partial_fluxes left for the
// partial cells.
TR_HD LineFace line_face(const Dims &D, const Geo &G, const SweepIn &S, int ax, const LineStep &s, const double *d,
                         const double *c, const double *flo, const double *fhi, int q, int a, int b)
{
    const int n = D.len(ax);
    const size_t g = line_g(D, ax, q, a, b);
    const size_t st = ax == 0 ? 1 : ax == 1 ? (size_t)(D.I + 2) : (size_t)(D.I + 2) * (size_t)(D.J + 2);
    const double w = S.vel[g];
    const uint32_t wa = hi32(w) & 0x7fffffffu;
    const bool nan = wa > 0x7ff00000u || (wa == 0x7ff00000u && lo32(w) != 0);
    const bool wneg = (hi32(w) >> 31) != 0, wzero = (wa | lo32(w)) == 0;
    const bool up = (!wneg || wzero) && !nan, pos = !wneg && !wzero && !nan;   // w >= 0, w > 0
    const double wd = w * S.dtv, step = line_div(s, wd);
    LineFace f;
    f.d = s.d;
    f.v = f.qv = 0.0;
    if (q < n) {
        const bool down = ax == 2 ? up : pos;
        const size_t gu = down ? g : g + st;
        const double v = S.vfl[gu];
        if (is_one(v)) {   // 1*u*dt
            f.v = wd;
            f.qv = step;
        } else if (!is_plus_zero(v) || !is_finite(w)) {   // an empty cell sends a zero
            f.v = vof_flux_rare(v, w, S.dtv, (down ? fhi : flo) + gu);
            f.qv = line_div(s, f.v);
        }
    }
    if (q == 1 || q == n || (q == n - 1 && !up)) {
        f.l = ls_face_rare(D, G, S, d, c, q, a, b);
    } else {
        // PH(q) + half*(1 - step)*(PH(q+1) - PH(q-1))/(2 d) from below,
        // PH(q+1) - half*(1 + step)*(PH(q+2) - PH(q))/(2 d) from above
        const size_t g0 = up ? g : g + st;
        const double t = 1.0 - flip_if(step, !up);
        const double e = line_div2(s, s.half * t * (S.phi[g0 + st] - S.phi[g0 - st]));
        const double ls = S.phi[g0] + flip_if(e, !up);
        f.l = w * ls * S.dtv;
    }
    f.ql = line_div(s, f.l);
    return f;
}

// The VOF of line_update for a cell with liquid in it or in its fluxes.
TR_RARE double line_vof_rare(LineStep s, int m, int n, double v0, double qvl, double qvh, double um, double ug,
                             double dtv, bool later, double first, double du, double den)
{
    double tv = v0;
    if (m >= 2) tv = tv + qvl;
    if (m <= n - 1) tv = tv - qvh;
    if (m == 1) tv = tv + line_div(s, v0 * um * dtv);
    if (m == n) tv = tv - line_div(s, v0 * ug * dtv);
    if (!later) tv = divd(tv, den);
    else tv = tv + s.rate * first * du;
    if (tv <= VOFEPS) tv = 0.0;
    if (tv >= 1.0 - VOFEPS) tv = 1.0;
    return tv;
}
TR_RARE double wall_flux_rare(LineStep s, double u, double ls, double dtv) { return line_div(s, u * ls * dtv); }

// sweep_update from the faces lo (not read at m = 1) and hi; s: this cell's
// spacing; LATER: the second or third sweep of the sub-step.  An empty cell
// without VOF fluxes stays empty: its sum is a zero, which the clip makes +0.
template <bool LATER>
TR_HD void line_update(const Dims &D, const SweepIn &S, int ax, const LineStep &s, const LineFace &lo,
                       const LineFace &hi, int m, int a, int b, double &vf_out, double &ls_out)
{
    const int n = D.len(ax);
    const size_t g = line_g(D, ax, m, a, b);
    const size_t st = ax == 0 ? 1 : ax == 1 ? (size_t)(D.I + 2) : (size_t)(D.I + 2) * (size_t)(D.J + 2);
    const double ug = S.vel[g], um = S.vel[g - st], v0 = S.vfl[g];
    const bool same = same_bits(lo.d, s.d);
    const double du = ug - um;
    const double den = LATER ? 1.0 : 1.0 - s.rate * du;
    const double first = LATER ? S.vf_first[g] : 0.0;
    // finite rate and du (or den neither zero nor infinite): zeros stay zeros
    const bool tame = LATER ? is_finite(du) && is_finite(s.rate) : exp_of(den) != 0 && is_finite(den);
    if (is_zero(v0) && is_zero(first) && is_zero(hi.qv) && (m < 2 || is_zero(lo.v)) && tame && is_finite(ug) &&
        is_finite(um)) {
        vf_out = 0.0;
    } else {
        const double qvl = m < 2 ? 0.0 : same ? lo.qv : line_div(s, lo.v);
        vf_out = line_vof_rare(s, m, n, v0, qvl, hi.qv, um, ug, S.dtv, LATER, first, du, den);
    }
    // + low face - high face, in the order - high + low at m = 2; at the low
    // wall - high + the wall's flux
    double q1, q2;
    if (m >= 2) {
        const double qll = same ? lo.ql : line_div(s, lo.l), qlh = flip_if(hi.ql, true);
        q1 = m >= 3 ? qll : qlh;
        q2 = m >= 3 ? qlh : qll;
    } else {
        const size_t bw = (size_t)(a - 1) + (size_t)D.plane_lead(ax) * (size_t)(b - 1);
        TR_CHECK(bw < D.plane_size(ax), "wall plane");
        q1 = flip_if(hi.ql, true);
        q2 = wall_flux_rare(s, S.bc_vel[bw], S.bc_lvs[bw], S.dtv);
    }
    const double tl = S.phi[g] + q1 + q2;
    if (LATER) ls_out = tl + s.rate * S.ls_first[g] * du;
    else ls_out = divd(tl, den);
}

// ---- redistancing (Redistance_Levelset 1689-1889) ----------------------

TR_HD bool inside_rect(double d1, double d2, double r10, double r11, double r20, double r21)
{
    return r10 <= d1 && d1 <= r11 && r20 <= d2 && d2 <= r21;
}

// Iscutface (1929-1959): the plane crosses the face at `fp` normal to cas.
TR_HD bool cut_face(double fp, double nxx, double nyy, double nzz, double diss, double dx, double dy, double dz,
                    int cas)
{
    double p1, p2, p3, p4;
    if (cas == 1) {
        p1 = fp * nxx - 0.5 * dy * nyy - 0.5 * dz * nzz + diss;
        p2 = fp * nxx - 0.5 * dy * nyy + 0.5 * dz * nzz + diss;
        p3 = fp * nxx + 0.5 * dy * nyy + 0.5 * dz * nzz + diss;
        p4 = fp * nxx + 0.5 * dy * nyy - 0.5 * dz * nzz + diss;
    } else if (cas == 2) {
        p1 = -0.5 * dx * nxx + fp * nyy - 0.5 * dz * nzz + diss;
        p2 = -0.5 * dx * nxx + fp * nyy + 0.5 * dz * nzz + diss;
        p3 = 0.5 * dx * nxx + fp * nyy + 0.5 * dz * nzz + diss;
        p4 = 0.5 * dx * nxx + fp * nyy - 0.5 * dz * nzz + diss;
    } else {
        p1 = -0.5 * dx * nxx - 0.5 * dy * nyy + fp * nzz + diss;
        p2 = -0.5 * dx * nxx + 0.5 * dy * nyy + fp * nzz + diss;
        p3 = 0.5 * dx * nxx + 0.5 * dy * nyy + fp * nzz + diss;
        p4 = 0.5 * dx * nxx - 0.5 * dy * nyy + fp * nzz + diss;
    }
    return !(p1 * p2 >= 0.0 && p2 * p3 >= 0.0 && p3 * p4 >= 0.0 && p4 * p1 >= 0.0);
}

// Shortest_Point_2d (1961-2060) on the face normal to cas (1, 2, 3), whose
// coordinate the caller has set: writes the other two.  Its y-face case
// solves for x dividing by |nz|, as the reference does.
TR_HD void shortest_point_2d(double nx1, double ny1, double nz1, double dis1, int ii, int jj, int kk, int cas,
                             double dx, double dy, double dz, double &xs, double &ys, double &zs)
{
    const double epsi = 1.0e-30;
    // (u, v) are the face's two in-plane axes in the reference's order.
    const double nu1 = cas == 1 ? ny1 : nx1, nv1 = cas == 3 ? ny1 : nz1;
    const double du = cas == 1 ? dy : dx, dv = cas == 3 ? dy : dz;
    const int iu = cas == 1 ? jj : ii, iv = cas == 3 ? jj : kk;
    const double temp = sqrt(nu1 * nu1 + nv1 * nv1 + epsi * epsi);
    const double nuu = nu1 / temp, nvv = nv1 / temp, diss = dis1 / temp;
    const double dij1 = nuu * du * (double)iu + nvv * dv * (double)iv + diss;
    const double up = du * (double)iu - dij1 * nuu, vp = dv * (double)iv - dij1 * nvv;
    double us, vs;
    if (inside_rect(up, vp, -0.5 * du, 0.5 * du, -0.5 * dv, 0.5 * dv)) {
        us = up;
        vs = vp;
    } else {
        const double uoff = fmax(fabs(up) - 0.5 * du, 0.0), voff = fmax(fabs(vp) - 0.5 * dv, 0.0);
        const double ufc = sgn(up) * 0.5 * du, vfc = sgn(vp) * 0.5 * dv;
        if (uoff * fabs(nuu) > voff * fabs(nvv)) {
            us = ufc;
            vs = (diss + nuu * us) / (sgn(-nvv) * fmax(fabs(nvv), TOLPAR));
        } else {
            vs = vfc;
            const double div = cas == 2 ? fabs(nvv) : fabs(nuu);
            us = (diss + nvv * vs) / (sgn(-nuu) * fmax(div, TOLPAR));
        }
    }
    if (cas == 1) { ys = us; zs = vs; }
    else if (cas == 2) { xs = us; zs = vs; }
    else { xs = us; ys = vs; }
}

// The third case with several axes of equal weight: the reference goes through
// them all, each writing into the same point.
TR_RARE double band_ties_rare(double nxx, double nyy, double nzz, double diss, int ii, int jj, int kk, double dx,
                              double dy, double dz, double xp, double yp, double zp, double ax, double ay, double az)
{
    const double X = dx * (double)ii, Y = dy * (double)jj, Z = dz * (double)kk;
    const double fc[3] = {sgn(xp) * 0.5 * dx, sgn(yp) * 0.5 * dy, sgn(zp) * 0.5 * dz};
    const double nn[3] = {nxx, nyy, nzz};
    double s[3] = {0.0, 0.0, 0.0};
    const double w[3] = {ax, ay, az};
    for (int c = 0; c < 3; ++c) {
        const int o1 = c == 0 ? 1 : 0, o2 = c == 2 ? 1 : 2;
        if (!(w[c] >= w[o1] && w[c] >= w[o2])) continue;
        int cas;
        if (cut_face(fc[c], nxx, nyy, nzz, diss, dx, dy, dz, c + 1)) cas = c;
        else cas = w[o1] > w[o2] ? o1 : o2;
        s[cas] = fc[cas];
        shortest_point_2d(nxx, nyy, nzz, nn[cas] * s[cas] + diss, ii, jj, kk, cas + 1, dx, dy, dz, s[0], s[1], s[2]);
    }
    return sqrt((X - s[0]) * (X - s[0]) + (Y - s[1]) * (Y - s[1]) + (Z - s[2]) * (Z - s[2]));
}

// The distance Redistance_Levelset measures from the centre (ii, jj, kk)
// cells away to an interface cell's plane n.x + diss = 0 (diss from the
// cell centre; the interface cell's spacings): the facing boundary point
// when it lies across the plane from the target (`side` = phi there),
// else the foot of the perpendicular inside the cell, else the nearest
// point of the plane's trace on the face it leaves through.
TR_HD double band_distance(double nxx, double nyy, double nzz, double diss, int ii, int jj, int kk, double dx,
                           double dy, double dz, double side)
{
    const int l = ii < -1 ? -1 : ii > 1 ? 1 : ii;
    const int m = jj < -1 ? -1 : jj > 1 ? 1 : jj;
    const int n = kk < -1 ? -1 : kk > 1 ? 1 : kk;
    const double xv = dx * (double)l / 2.0, yv = dy * (double)m / 2.0, zv = dz * (double)n / 2.0;
    const double dv = nxx * xv + nyy * yv + nzz * zv + diss;
    const double X = dx * (double)ii, Y = dy * (double)jj, Z = dz * (double)kk;
    if (dv * sgn(side) <= 0.0) return sqrt((X - xv) * (X - xv) + (Y - yv) * (Y - yv) + (Z - zv) * (Z - zv));
    const double dij1 = nxx * dx * (double)ii + nyy * dy * (double)jj + nzz * dz * (double)kk + diss;
    const double xp = X - dij1 * nxx, yp = Y - dij1 * nyy, zp = Z - dij1 * nzz;
    if (-0.5 * dx <= xp && xp <= 0.5 * dx && -0.5 * dy <= yp && yp <= 0.5 * dy && -0.5 * dz <= zp && zp <= 0.5 * dz)
        return sqrt((X - xp) * (X - xp) + (Y - yp) * (Y - yp) + (Z - zp) * (Z - zp));
    const double ax = fmax(fabs(xp) - 0.5 * dx, 0.0) * fabs(nxx);
    const double ay = fmax(fabs(yp) - 0.5 * dy, 0.0) * fabs(nyy);
    const double az = fmax(fabs(zp) - 0.5 * dz, 0.0) * fabs(nzz);
    // One axis outweighs the others (almost always): its face, one copy of the
    // work for all three axes, so that a warp's lanes stay together.
    const int c = ay > ax ? (az > ay ? 2 : 1) : (az > ax ? 2 : 0);
    const double wc = c == 0 ? ax : c == 1 ? ay : az;
    const double w1 = c == 0 ? ay : ax, w2 = c == 2 ? ay : az;
    if (!(wc > w1 && wc > w2))
        return band_ties_rare(nxx, nyy, nzz, diss, ii, jj, kk, dx, dy, dz, xp, yp, zp, ax, ay, az);
    const double nc = c == 0 ? nxx : c == 1 ? nyy : nzz;
    const double f = sgn(c == 0 ? xp : c == 1 ? yp : zp) * 0.5 * (c == 0 ? dx : c == 1 ? dy : dz);
    // cut_face: the corner sums in the order x, y, z (the face's own term is the
    // first or second addend on the x and y faces, the third on the z face)
    const double ha = 0.5 * (c == 0 ? dy : dx) * (c == 0 ? nyy : nxx), hb = 0.5 * (c == 2 ? dy : dz) * (c == 2 ? nyy : nzz);
    const double fn = f * nc;
    const bool zc = c == 2;
    const double p1 = (zc ? -ha - hb : fn - ha) + (zc ? fn : -hb) + diss;
    const double p2 = (zc ? -ha + hb : fn - ha) + (zc ? fn : hb) + diss;
    const double p3 = (zc ? ha + hb : fn + ha) + (zc ? fn : hb) + diss;
    const double p4 = (zc ? ha - hb : fn + ha) + (zc ? fn : -hb) + diss;
    int cas = c;
    if (p1 * p2 >= 0.0 && p2 * p3 >= 0.0 && p3 * p4 >= 0.0 && p4 * p1 >= 0.0)
        cas = w1 > w2 ? (c == 0 ? 1 : 0) : (c == 2 ? 1 : 2);
    const double fs = cas == c ? f : sgn(cas == 0 ? xp : cas == 1 ? yp : zp) * 0.5 * (cas == 0 ? dx : cas == 1 ? dy : dz);
    double s0 = fs, s1 = fs, s2 = fs;   // the face's coordinate; the other two are set
    const double ns = cas == 0 ? nxx : cas == 1 ? nyy : nzz;
    shortest_point_2d(nxx, nyy, nzz, ns * fs + diss, ii, jj, kk, cas + 1, dx, dy, dz, s0, s1, s2);
    return sqrt((X - s0) * (X - s0) + (Y - s1) * (Y - s1) + (Z - s2) * (Z - s2));
}

// ---- FP32 bounds of a band distance ----------------------------------------
//
// Only the least distance of each target counts, so a pair whose FP32 lower
// bound exceeds the target's least FP32 upper bound needs no FP64 work.  The
// bounds come from band_distance's steps in FP32 on lengths scaled by the
// cell's largest spacing, with every comparison required to hold by more than
// the error of its two sides; a pair that comes too close to any of them has
// no bounds and is computed.  Errors (in units of the scale, u = 2^-24): the
// inputs carry a few u each, |X| <= 4 per axis, |dis| <= 2 and |n| <= 1 give
// at most 8e-6 for dv, dij1 and the foot point; BE1 doubles that.

struct BandSource {
    float n[3], dis, d[3], h;
    bool ok;   // inside the range the error bounds hold for
};
// What Iscutface and Shortest_Point_2d form of one face of the cell (index
// 2 * axis + (1 on the high side)), whatever the target: u, v are its in-plane
// axes.  inv_v = -1/nv and inv_u = 1/(-nu) -- on a y face over |nz| -- or 0
// where the quotient is too steep to bound.
struct BandFace {
    float nu, nv, ds, e4, e5, inv_u, inv_v;
    int cut;   // 1: the plane crosses the face, 0: it does not, -1: FP32 cannot tell
};

constexpr float BE1 = 1.6e-5f;

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float band_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float band_sqrt(float a)   // within 2^-23 relative
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
#else
TR_HD float band_fma(float a, float b, float c) { return fmaf(a, b, c); }
#if !defined(TR_SQRT_ERROR)
#define TR_SQRT_ERROR 0.0   // host checks: the approximate square root's relative error
#endif
TR_HD float band_sqrt(float a) { return (float)((double)sqrtf(a) * (1.0 + TR_SQRT_ERROR)); }
#endif

// v[q] by selects: the arrays stay in registers.
template <typename T>
TR_HD T pick(const T (&v)[3], int q) { return q == 0 ? v[0] : q == 1 ? v[1] : v[2]; }

// From the FP32 values of an interface cell's normal, centre distance and
// spacings.
TR_HD BandSource band_source(float n1, float n2, float n3, float dis, float dx, float dy, float dz)
{
    BandSource s;
    s.n[0] = n1; s.n[1] = n2; s.n[2] = n3;
    const float m = dx > dy ? dx : dy;
    s.h = m > dz ? m : dz;
    s.d[0] = dx / s.h; s.d[1] = dy / s.h; s.d[2] = dz / s.h;
    s.dis = dis / s.h;
    s.ok = s.h > 1e-15f && s.h < 1e15f && s.d[0] > 1e-3f && s.d[1] > 1e-3f && s.d[2] > 1e-3f &&
           fabsf(s.dis) <= 2.0f && n1 * n1 + n2 * n2 + n3 * n3 <= 1.001f;
    return s;
}

TR_HD BandFace band_face(const BandSource &B, int face)
{
    const int c = face >> 1, u = c == 0 ? 1 : 0, v = c == 2 ? 1 : 2;
    const float n = pick(B.n, c), pu = pick(B.n, u), pv = pick(B.n, v);
    const float base = (face & 1 ? 0.5f : -0.5f) * pick(B.d, c) * n + B.dis;
    BandFace f;
    const float h1 = 0.5f * pick(B.d, u) * pu, h2 = 0.5f * pick(B.d, v) * pv;
    const float p1 = base - h1 - h2, p2 = base - h1 + h2, p3 = base + h1 + h2, p4 = base + h1 - h2;
    f.cut = (p1 > 0.f) == (p2 > 0.f) && (p2 > 0.f) == (p3 > 0.f) && (p3 > 0.f) == (p4 > 0.f) ? 0 : 1;
    if (!(fabsf(p1) > BE1 && fabsf(p2) > BE1 && fabsf(p3) > BE1 && fabsf(p4) > BE1)) f.cut = -1;
    const float t = sqrtf(pu * pu + pv * pv);
    f.nu = f.nv = f.ds = f.e5 = f.inv_u = f.inv_v = 0.f;
    f.e4 = 1e30f;   // no bounds: every comparison comes too close
    if (t > 0.02f) {
        const float r = 1.0f / t;
        f.nu = pu * r;
        f.nv = pv * r;
        f.ds = base * r;
        f.e4 = 2.4e-5f + 1.0e-5f * r;
        f.e5 = 6.0e-6f * r + 6.0e-6f;
        if (fabsf(f.nv) > 0.02f) f.inv_v = -1.0f / f.nv;
        const float div = c == 1 ? fabsf(f.nv) : fabsf(f.nu);
        if (div > 0.02f && fabsf(f.nu) > 1.0e-5f) f.inv_u = 1.0f / copysignf(div, -f.nu);
    }
    return f;
}

// v is certainly inside [-half, half], certainly outside, or neither (0).
TR_HD int band_side(float v, float half, float e) { return fabsf(v) < half - e ? 1 : fabsf(v) > half + e ? -1 : 0; }

// Bounds of band_distance for the offset (ii, jj, kk) and the sign of the
// level set there; false when FP32 cannot decide.  F: the cell's six faces.
TR_HD bool band_bounds(const BandSource &B, const BandFace *F, int ii, int jj, int kk, bool neg, float &lo, float &hi)
{
    if (!B.ok) return false;
    const int o[3] = {ii, jj, kk};
    float X[3], t[3], dv = B.dis, dij = B.dis;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int l = o[q] < -1 ? -1 : o[q] > 1 ? 1 : o[q];
        X[q] = B.d[q] * (float)o[q];
        t[q] = B.d[q] * (0.5f * (float)l);   // the facing boundary point
        dv = band_fma(B.n[q], t[q], dv);
        dij = band_fma(B.n[q], X[q], dij);
    }
    const float sdv = neg ? -dv : dv;
    if (!(fabsf(sdv) > BE1)) return false;
    float a0, a1, a2, err;   // target minus the nearest point
    if (sdv < 0.f) {
        a0 = X[0] - t[0]; a1 = X[1] - t[1]; a2 = X[2] - t[2];
        err = BE1;
    } else {
        float xp[3], w[3];
        int in[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            xp[q] = band_fma(-dij, B.n[q], X[q]);
            in[q] = band_side(xp[q], 0.5f * B.d[q], BE1);
            // a coordinate inside weighs exactly 0
            w[q] = in[q] > 0 ? 0.f : (fabsf(xp[q]) - 0.5f * B.d[q]) * fabsf(B.n[q]);
        }
        if (in[0] == 0 || in[1] == 0 || in[2] == 0) return false;
        if (in[0] > 0 && in[1] > 0 && in[2] > 0) {
            a0 = X[0] - xp[0]; a1 = X[1] - xp[1]; a2 = X[2] - xp[2];
            err = 2.0f * BE1;
        } else {
            // the face the foot point leaves through: the largest weight, which
            // must be so beyond doubt
            int c = w[1] > w[0] ? 1 : 0;
            if (w[2] > pick(w, c)) c = 2;
            const int o1 = c == 0 ? 1 : 0, o2 = c == 2 ? 1 : 2;
            const float wc = pick(w, c) - 2.0f * BE1, w1 = pick(w, o1), w2 = pick(w, o2);
            if (!(wc > w1) || !(wc > w2)) return false;
            int face = 2 * c + (pick(xp, c) > 0.f ? 1 : 0);
            const int cut = F[face].cut;
            if (cut < 0) return false;
            if (cut == 0) {   // the other axis that weighs more, the second if neither does
                if (!(w1 == 0.f && w2 == 0.f) && !(fabsf(w1 - w2) > 2.0f * BE1)) return false;
                const int cas = w1 > w2 ? o1 : o2;
                const float x = pick(xp, cas);
                if (!(fabsf(x) > BE1)) return false;
                face = 2 * cas + (x > 0.f ? 1 : 0);
            }
            // Shortest_Point_2d on that face
            const BandFace f = F[face];
            const int cas = face >> 1, u = cas == 0 ? 1 : 0, v = cas == 2 ? 1 : 2;
            const float Xu = pick(X, u), Xv = pick(X, v);
            const float dj = band_fma(f.nu, Xu, band_fma(f.nv, Xv, f.ds));
            const float up = band_fma(-dj, f.nu, Xu), vp = band_fma(-dj, f.nv, Xv);
            const float hu = 0.5f * pick(B.d, u), hv = 0.5f * pick(B.d, v);
            const int iu = band_side(up, hu, f.e4), iv = band_side(vp, hv, f.e4);
            if (iu == 0 || iv == 0) return false;
            float us = up, vs = vp;
            err = 2.0f * f.e4 + BE1;
            if (iu < 0 || iv < 0) {
                const float wu = iu > 0 ? 0.f : (fabsf(up) - hu) * fabsf(f.nu);
                const float wv = iv > 0 ? 0.f : (fabsf(vp) - hv) * fabsf(f.nv);
                if (!(fabsf(wu - wv) > 2.0f * f.e4)) return false;
                float inv, s;
                if (wu > wv) {
                    us = copysignf(hu, up);
                    inv = f.inv_v;
                    s = vs = band_fma(f.nu, us, f.ds) * inv;
                } else {
                    vs = copysignf(hv, vp);
                    inv = f.inv_u;
                    s = us = band_fma(f.nv, vs, f.ds) * inv;
                }
                if (inv == 0.f) return false;
                err = f.e5 * fabsf(inv) + 2.0e-6f * fabsf(s) + f.e4 + BE1;
            }
            a0 = pick(X, cas) - (face & 1 ? 0.5f : -0.5f) * pick(B.d, cas);
            a1 = Xu - us;
            a2 = Xv - vs;
        }
    }
    const float dist = band_sqrt(band_fma(a0, a0, band_fma(a1, a1, a2 * a2)));
    err = band_fma(2.0e-6f, dist, err);
    lo = (dist - err) * B.h;
    hi = (dist + err) * B.h;
    return true;
}

// An upper bound of every cell's initial key (1e4).
constexpr float BAND_UB = 1.001e4f;

TR_HD bool band_interface(double v) { return 0.0 + 1.0e-15 < v && v < 1.0 - 1.0e-15; }
TR_HD bool band_target(double v) { return v < 0.0 + 1.0e-15 || v > 1.0 - 1.0e-15; }

// The bits of a non-negative double order like the double.
TR_HD uint64_t key_of(double v) { return bits_of(v); }
TR_HD double value_of(uint64_t u) { return from_bits(u); }

TR_HD void atomic_min_key(unsigned long long *slot, unsigned long long key)
{
#if defined(__CUDA_ARCH__)
    atomicMin(slot, key);
#else
    if (key < *slot) *slot = key;
#endif
}

constexpr int BAND_SPAN = 2 * BAND + 1;
constexpr int BAND_CELLS = BAND_SPAN * BAND_SPAN * BAND_SPAN;   // 729 offsets

// Offset t (0 .. BAND_CELLS-1) of an interface cell's band, ii fastest.
TR_HD void band_offset(int t, int &ii, int &jj, int &kk)
{
    ii = t % BAND_SPAN - BAND;
    jj = (t / BAND_SPAN) % BAND_SPAN - BAND;
    kk = t / (BAND_SPAN * BAND_SPAN) - BAND;
}

// Interior cell of index c (i fastest), the inverse of Dims::n, in 32-bit
// arithmetic (the transport context holds fewer than 2^32 interior cells).
TR_HD void cell_of(const Dims &D, uint32_t c, int &i, int &j, int &k)
{
    const uint32_t r = c / (uint32_t)D.I;
    i = (int)(c - r * (uint32_t)D.I) + 1;
    const uint32_t kq = r / (uint32_t)D.J;
    j = (int)(r - kq * (uint32_t)D.J) + 1;
    k = (int)kq + 1;
}

// One pair of the band (1726-1861): the interface cell (i, j, k) and its
// offset t.  A full or empty target cell within BAND cells in each index is
// marked and keeps the least distance seen; dis holds the distances from
// the cell centres.  The minimum does not depend on the order of the pairs.
TR_HD void band_pair(const Dims &D, const Geo &G, const double *vfl, const double *phi, const double *nx,
                     const double *ny, const double *nz, const double *dis, int i, int j, int k, int t,
                     unsigned long long *key, uint8_t *fix)
{
    int ii, jj, kk;
    band_offset(t, ii, jj, kk);
    const int ti = i + ii, tj = j + jj, tk = k + kk;
    if (!(1 <= ti && ti <= D.I && 1 <= tj && tj <= D.J && 1 <= tk && tk <= D.K)) return;
    const size_t tg = D.g(ti, tj, tk), tc = D.n(ti, tj, tk);
    if (!band_target(vfl[tg])) return;
    const size_t g = D.g(i, j, k), c = D.n(i, j, k);
    fix[tc] = 1;
    const double deuc = band_distance(nx[g], ny[g], nz[g], dis[g], ii, jj, kk, G.dx[c], G.dy[c], G.dz[c], phi[tg]);
    atomic_min_key(key + tc, key_of(deuc));
}

// One interface cell's whole band, pair by pair.
TR_HD void band_scatter(const Dims &D, const Geo &G, const double *vfl, const double *phi, const double *nx,
                        const double *ny, const double *nz, const double *dis, int i, int j, int k,
                        unsigned long long *key, uint8_t *fix)
{
    if (!band_interface(vfl[D.g(i, j, k)])) return;
    for (int t = 0; t < BAND_CELLS; ++t) band_pair(D, G, vfl, phi, nx, ny, nz, dis, i, j, k, t, key, fix);
}

TR_RARE double band_value_rare(double v, double dx, const double *dis, bool fixed, unsigned long long key)
{
    if (band_interface(v)) return sgn(0.5 - v) * fabs(*dis);
    if (fixed) return sgn(0.5 - v) * value_of(key);
    return (double)(BAND + 1) * dx * sqrt(3.0) * sgn(0.5 - v);
}

// The level set each cell ends with (1866-1882).
TR_HD double band_value(const Dims &D, const Geo &G, const double *vfl, const double *dis, int i, int j, int k,
                        const unsigned long long *key, const uint8_t *fix)
{
    const size_t g = D.g(i, j, k), c = D.n(i, j, k);
    const double v = vfl[g];
    if (is_plus_zero(v) || is_one(v)) {   // empty or full: only the sign depends on v
        const double m = fix[c] ? value_of(key[c]) : (double)(BAND + 1) * G.dx[c] * sqrt(3.0);
        return flip_if(m, hi32(v) != 0);
    }
    return band_value_rare(v, G.dx[c], dis + g, fix[c] != 0, key[c]);
}

// ---- boundary planes (BoundaryConditionLvsVof 2087-2221) -----------------

struct WallIn {
    double *phil, *vofl;                     // ghosted: the sub-step's result
    double *phil_more[2], *vofl_more[2];     // the other ping-pong buffers, whose
                                             // ghost faces must match (or null)
    const double *nxl;                       // liquid normal, ghosted
    const double *nx, *ny, *nz;              // fluid normals, ghosted
    double *lvs_bc[6], *vof_bc[6];           // planes W, E, S, N, B, T
    int lvs_flag[6], vof_flag[6];
    double lvs_const[6], vof_const[6];
};

TR_HD double typical_bc(int flag, double cst, double var, double d) { return flag == 0 ? cst : var - cst * d / 2.0; }

// Point t of the wall planes normal to `axis`, both faces, level set then
// VOF.  W and E level-set planes are phiL -/+ nxL*dx/2 (the reference hands
// BCLvsW/E the liquid normals); the others are TypicalBC; the level-set
// ghosts step by the fluid normal times the spacing, the north one
// subtracting like the south; the VOF ghosts copy the wall cell.
TR_HD void wall_point(const Dims &D, const Geo &G, const WallIn &W, int axis, size_t t)
{
    const int lead = D.plane_lead(axis);
    const int a = (int)(t % (size_t)lead) + 1, b = (int)(t / (size_t)lead) + 1;
    const int n = D.len(axis);
    const size_t g1 = line_g(D, axis, 1, a, b), gn = line_g(D, axis, n, a, b);
    const size_t g0 = line_g(D, axis, 0, a, b), gx = line_g(D, axis, n + 1, a, b);
    const size_t c1 = line_n(D, axis, 1, a, b), cn = line_n(D, axis, n, a, b);
    const double *d = axis == 0 ? G.dx : axis == 1 ? G.dy : G.dz;
    const double *fn = axis == 0 ? W.nx : axis == 1 ? W.ny : W.nz;
    const double d1 = d[c1], dn = d[cn];
    const int lo = 2 * axis, hi = 2 * axis + 1;
    // level set
    double p1 = W.phil[g1], pn = W.phil[gn];
    double wlo = typical_bc(W.lvs_flag[lo], W.lvs_const[lo], p1, d1);
    double whi = typical_bc(W.lvs_flag[hi], W.lvs_const[hi], pn, -dn);
    if (axis == 0) {
        wlo = p1 - W.nxl[g1] * d1 / 2.0;
        whi = pn - W.nxl[gn] * (-dn) / 2.0;
    }
    W.lvs_bc[lo][t] = wlo;
    W.lvs_bc[hi][t] = whi;
    const double lo_ghost = p1 - fn[g1] * d1;
    const double hi_ghost = axis == 1 ? pn - fn[gn] * dn : pn + fn[gn] * dn;
    W.phil[g0] = lo_ghost;
    W.phil[gx] = hi_ghost;
    // VOF
    const double v1 = W.vofl[g1], vn = W.vofl[gn];
    W.vof_bc[lo][t] = typical_bc(W.vof_flag[lo], W.vof_const[lo], v1, d1);
    W.vof_bc[hi][t] = typical_bc(W.vof_flag[hi], W.vof_const[hi], vn, -dn);
    W.vofl[g0] = v1;
    W.vofl[gx] = vn;
    for (int q = 0; q < 2; ++q) {
        if (W.phil_more[q]) {
            W.phil_more[q][g0] = lo_ghost;
            W.phil_more[q][gx] = hi_ghost;
        }
        if (W.vofl_more[q]) {
            W.vofl_more[q][g0] = v1;
            W.vofl_more[q][gx] = vn;
        }
    }
}

// ---- the velocity cells' liquid fields (ComputeUVWLiquidField 174-353) ----

// ConvertTheCoordinateSystem (2458-2465): phi measured from the corner.
TR_HD double corner_level(double dx, double dy, double dz, double nx, double ny, double nz, double phi)
{
    return phi + 0.5 * (fabs(nx) * dx + fabs(ny) * dy + fabs(nz) * dz);
}

// The four averaged fields (phiL, nxL, nyL, nzL) of velocity family `fam`
// (0 U, 1 V, 2 W) at its cell (p, q, r), 0 <= p < I, 0 <= q < J, 0 <= r < K.
// DirectionAverageArray (328-353) writes the average of the P cells
// (i, i+1) along the family's axis into VelCell(i-1, j-1, k-1) -- an
// assumed-shape dummy numbered from 1 over arrays allocated from 0 -- and
// copies the last one once more, so the cell gathers the P pair at
// (p+1, q+1, r+1) with the axis index held at n-1.  d: the P spacing along
// the axis.
TR_HD void family_average(const Dims &D, int fam, const double *d, const double *const pin[4], int p, int q, int r,
                          double out[4])
{
    int i = p + 1, j = q + 1, k = r + 1;
    if (fam == 0 && i == D.I) i = D.I - 1;
    if (fam == 1 && j == D.J) j = D.J - 1;
    if (fam == 2 && k == D.K) k = D.K - 1;
    const int i2 = i + (fam == 0), j2 = j + (fam == 1), k2 = k + (fam == 2);
    const double lamda = divd(d[D.n(i2, j2, k2)], d[D.n(i, j, k)] + d[D.n(i2, j2, k2)]);
    const size_t a = D.g(i, j, k), b = D.g(i2, j2, k2);
    for (int f = 0; f < 4; ++f) out[f] = lamda * pin[f][a] + (1.0 - lamda) * pin[f][b];
}

// The liquid fraction of velocity cell (i, j, k) of family `fam`: the
// liquid in the half of P cell (i, j, k) on its high side plus the half of
// the next P cell on its low side, over the velocity cell's volume; the
// last cell of each line takes the P cell's own fraction (ComputeUVW-
// LiquidField 186-297).  Kept as the reference computes them: the V cell's
// low half cuts with the whole dy and the unshifted level set, its high
// half starts from phiL(i,j,k) with the normal of (i,j+1,k); the W cell's
// high half shifts by +dz/2 where the U cell's shifts by -dx/2.
TR_HD double family_vofl(const Dims &D, int fam, const double *pdx, const double *pdy, const double *pdz,
                         const double *phil, const double *nxl, const double *nyl, const double *nzl,
                         const double *vofl, const double *vdx, const double *vdy, const double *vdz, int i, int j,
                         int k)
{
    const int n = D.len(fam), m = fam == 0 ? i : fam == 1 ? j : k;
    const size_t a = D.g(i, j, k), na = D.n(i, j, k);
    if (m == n) return vofl[a];
    const int i2 = i + (fam == 0), j2 = j + (fam == 1), k2 = k + (fam == 2);
    const size_t b = D.g(i2, j2, k2), nb = D.n(i2, j2, k2);
    double dcell, phinew, dist, left, right;
    if (fam == 0) {
        dcell = pdx[na] / 2.0;
        phinew = phil[a] + dcell * nxl[a];
        dist = corner_level(dcell, pdy[na], pdz[na], nxl[a], nyl[a], nzl[a], phinew);
        left = volume_fraction(dcell, pdy[na], pdz[na], nxl[a], nyl[a], nzl[a], dist);
        left = dcell * pdy[na] * pdz[na] - left;
        dcell = pdx[nb] / 2.0;
        phinew = phil[b] - dcell * nxl[b];
        dist = corner_level(dcell, pdy[nb], pdz[nb], nxl[b], nyl[b], nzl[b], phinew);
        right = volume_fraction(dcell, pdy[nb], pdz[nb], nxl[b], nyl[b], nzl[b], dist);
        right = dcell * pdy[nb] * pdz[nb] - right;
    } else if (fam == 1) {
        dcell = pdy[na] / 2.0;
        dist = corner_level(pdx[na], pdy[na], pdz[na], nxl[a], nyl[a], nzl[a], phil[a]);
        left = volume_fraction(pdx[na], dcell, pdz[na], nxl[a], nyl[a], nzl[a], dist);
        left = pdx[na] * dcell * pdz[na] - left;
        dcell = pdy[nb] / 2.0;
        phinew = phil[a] + dcell * nyl[b];
        dist = corner_level(pdx[nb], dcell, pdz[nb], nxl[b], nyl[b], nzl[b], phinew);
        right = volume_fraction(pdx[nb], dcell, pdz[nb], nxl[b], nyl[b], nzl[b], dist);
        right = pdx[nb] * dcell * pdz[nb] - right;
    } else {
        dcell = pdz[na] / 2.0;
        phinew = phil[a] + dcell * nzl[a];
        dist = corner_level(pdx[na], pdy[na], dcell, nxl[a], nyl[a], nzl[a], phinew);
        left = volume_fraction(pdx[na], pdy[na], dcell, nxl[a], nyl[a], nzl[a], dist);
        left = pdx[na] * pdy[na] * dcell - left;
        dcell = pdz[nb] / 2.0;
        phinew = phil[b] + dcell * nzl[b];
        dist = corner_level(pdx[nb], pdy[nb], dcell, nxl[b], nyl[b], nzl[b], phinew);
        right = volume_fraction(pdx[nb], pdy[nb], dcell, nxl[b], nyl[b], nzl[b], dist);
        right = pdx[nb] * pdy[nb] * dcell - right;
    }
    return divd(divd(divd(left + right, vdx[na]), vdy[na]), vdz[na]);
}

}  // namespace tr
