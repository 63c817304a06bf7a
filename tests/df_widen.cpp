// df_widen.cpp -- the double-float to FP64 conversion of
// simcoflow3d_gb300/csrc/scf_df.cuh against the FP64 addition, its device
// intrinsics restated for the host.  Test infrastructure.
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
struct float2 { float x, y; };
static inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline int __float2int_rn(float f)
{
    if (std::isnan(f)) return 0;
    return f >= 2147483648.f ? INT_MAX : f < -2147483648.f ? INT_MIN : (int)std::nearbyintf(f);
}
static inline double __hiloint2double(int hi, int lo)
{
    const uint64_t b = ((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}
#include "scf_df.cuh"

// mode 0: any exponent, lo of 24 to 64 binary orders below hi; 1: ties and
// short significands, powers of two; 2: zeros, subnormals, infinities, pairs
// that are not normalised.  Returns the number of results that differ.
extern "C" long check_widen(unsigned seed, long n, int mode)
{
    std::mt19937_64 g(seed);
    long bad = 0;
    for (long s = 0; s < n; ++s) {
        const uint64_t r = g(), q = g();
        unsigned u = (unsigned)(r & 0x807fffffu) | (1u + (unsigned)((r >> 32) % 254)) << 23;
        if (mode == 1) u &= ~0u << (q >> 8) % 24;
        if (mode == 2 && q % 3 == 0) u &= q % 2 ? 0x807fffffu : 0x80000000u;
        if (mode == 2 && q % 17 == 0) u = 0x7f800000u;
        const float hi = __uint_as_float(u);
        float lo = std::ldexp(std::fabs(hi), -24 - (int)((q >> 16) % 40)) * (1.f + (float)(q >> 32 & 0x7fffff) * 0x1p-23f);
        if (mode == 1) lo = __uint_as_float(__float_as_uint(lo) & ~0u << (q >> 24) % 24);
        const float half = (std::nextafterf(std::fabs(hi), INFINITY) - std::fabs(hi)) * 0.5f;
        if (mode < 2 && std::isfinite(half) && lo > half) lo = half;
        if (mode == 2 && q % 5 == 0) lo = hi * (float)(q % 7);
        if (mode == 2 && q % 11 == 0) lo = 0.f;
        if (q >> 63) lo = -lo;
        const double ref = (double)hi + (double)lo, got = dwide(float2{hi, lo});
        if (std::isnan(ref) ? !std::isnan(got) : std::memcmp(&ref, &got, 8) != 0) ++bad;
    }
    return bad;
}
