// scf_df.cuh -- FP32 and double-float values to FP64 without the FP64 pipe.
#pragma once

// FP32 -> FP64 widening on the integer pipe (exact: the exponent is rebiased
// and the significand shifted into place).  Zeros keep their sign; the rare
// subnormal inputs, Inf and NaN take the hardware conversion.
__device__ __forceinline__ double widen(float f)
{
    const unsigned u = __float_as_uint(f);
    const unsigned e = (u >> 23) & 0xffu;
    if (e - 1u < 254u) {   // normal numbers
        const unsigned hi = (u & 0x80000000u) | ((e + 896u) << 20) | ((u & 0x7fffffu) >> 3);
        return __hiloint2double((int)hi, (int)(u << 29));
    }
    if ((u & 0x7fffffffu) == 0u) return __hiloint2double((int)(u & 0x80000000u), 0);
    return (double)f;
}
// The FP64 value hi + lo of a double-float (|lo| <= ulp(hi) / 2), rounded as
// the FP64 addition rounds it, on the integer and FP32 pipes.  hi widened has
// 29 zero bits at its end, so the sum is hi's bits plus lo in units of hi's
// FP64 ulp, rounded to the nearest even integer: the scaling is by a power of
// two, and an even hi leaves the tie rule to the conversion.  Small exponents
// (the scale's or lo's would leave FP32's range), Inf, NaN and powers of two
// (a borrow there halves the ulp) and pairs that are not normalised take the
// FP64 addition, out of line so that it is not executed under a predicate.
// An FP64 warp instruction holds its pipe for 16 cycles: the (r, z) product at
// 256^3 took 79 us with one for this and one for the product, 67 without (48
// with its loads in flight); k_spmv_df 172 -> 166.
__device__ __noinline__ double dwide_add(float hi, float lo) { return widen(hi) + widen(lo); }
__device__ __forceinline__ double dwide(float2 x)
{
    const unsigned u = __float_as_uint(x.x), e = (u >> 23) & 0xffu, neg = (unsigned)((int)u >> 31);
    if (((u | __float_as_uint(x.y)) & 0x7fffffffu) == 0u)
        return __hiloint2double((int)(u & __float_as_uint(x.y) & 0x80000000u), 0);
    if (e - 64u >= 191u || (u & 0x7fffffu) == 0u) return dwide_add(x.x, x.y);
    const int l = __float2int_rn(__fmul_rn(x.y, __uint_as_float((306u - e) << 23)));   // lo 2^(179 - e)
    if ((unsigned)l + 0x10000000u > 0x20000000u) return dwide_add(x.x, x.y);
    const int d = (l ^ (int)neg) - (int)neg;                                           // towards |hi|
    const unsigned h = (u & 0x80000000u) | ((e + 896u) << 20) | ((u & 0x7fffffu) >> 3), lw = u << 29;
    const unsigned lo = lw + (unsigned)d;
    return __hiloint2double((int)(h + (unsigned)(d >> 31) + (lo < lw ? 1u : 0u)), (int)lo);
}
