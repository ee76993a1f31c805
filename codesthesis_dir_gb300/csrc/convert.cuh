// Conversions between float and double without FP64 instructions.
#pragma once

#include <cuda_runtime.h>

// Conversions between float and double on the integer pipe.  GB300 issues
// FP64 instructions (conversions included) at about 1/64 of the FP32 rate,
// and the defect-correction loop converts every point twice per outer
// iteration.  Both functions round as IEEE 754 binary conversion does
// (round to nearest, ties to even; float -> double is exact) over the whole
// range, denormals, infinities and overflow included, with integer
// operations only, so that no FP64 instruction is issued even on a
// predicated path.  A NaN converts to a quiet NaN of the same sign.
// gb_check_conversions compares both with the hardware conversions.
__device__ __forceinline__ float d2f_rn(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned int sign = (unsigned int)(b >> 32) & 0x80000000u;
    const int e = (int)((b >> 52) & 0x7ffu);
    const unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    unsigned int r;
    if (e >= 897 && e <= 1150) {
        // normal float range: keep the top 23 fraction bits, round on the
        // 29 dropped (a carry into the exponent rounds up to the next
        // binade, or to infinity past the largest float)
        r = ((unsigned int)(e - 896) << 23) | (unsigned int)(m >> 29);
        const unsigned int rem = (unsigned int)(m & 0x1FFFFFFFull);
        r += (rem > 0x10000000u || (rem == 0x10000000u && (r & 1u))) ? 1u : 0u;
    } else if (e == 0x7ff) {
        r = m ? 0x7fc00000u : 0x7f800000u;
    } else if (e > 1150) {
        r = 0x7f800000u;   // at or above 2^128: overflows to infinity
    } else if (e == 0) {
        r = 0u;            // double denormals are far below the float range
    } else {
        // float denormal range: the result counts units of 2^-149, the
        // significand (with its hidden bit) shifted right by 926 - e >= 30
        const int sh = 926 - e;
        if (sh > 53) {
            r = 0u;        // below half the smallest denormal
        } else {
            const unsigned long long full = m | (1ull << 52);
            r = (unsigned int)(full >> sh);
            const unsigned long long rem = full & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
            r += (rem > half || (rem == half && (r & 1u))) ? 1u : 0u;
        }
    }
    return __uint_as_float(sign | r);
}

__device__ __forceinline__ double f2d(float v)
{
    const unsigned int u = __float_as_uint(v);
    const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
    const unsigned int e = (u >> 23) & 0xffu, m = u & 0x7FFFFFu;
    unsigned long long r;
    if (e != 0u && e != 255u) {
        r = ((unsigned long long)(e + 896u) << 52) | ((unsigned long long)m << 29);
    } else if (e == 255u) {
        r = m ? 0x7ff8000000000000ull | ((unsigned long long)m << 29) : 0x7ff0000000000000ull;
    } else if (m == 0u) {
        r = 0ull;
    } else {
        // float denormal m * 2^-149: normalise so that the leading bit of m
        // becomes the hidden bit
        const int lz = __clz(m) - 8;   // m < 2^23: 9 or more leading zeros
        r = ((unsigned long long)(897 - lz) << 52) | ((unsigned long long)((m << lz) & 0x7FFFFFu) << 29);
    }
    return __longlong_as_double((long long)(sign | r));
}
