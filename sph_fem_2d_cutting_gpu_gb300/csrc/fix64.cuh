// fix64.cuh -- FP64-accurate arithmetic on the integer pipes.
//
// GB300 executes two FP64 operations per SM and clock: one FP64 instruction
// occupies its pipe for as long as a scheduler issues 64 others.  The kernels
// bound by that pipe form the parts of an expression that are products,
// quotients and polynomials of known sign here, on 64-bit integer mantissas: a
// product is three 32 x 32 -> 64-bit multiplications, and 64 mantissa bits
// through a chain keep its error below the one rounding of its last step.
// A value is m * 2^e with an unsigned 64-bit m.
#pragma once

#include "common.cuh"

namespace sphfem {

struct Fix64 {
    uint64_t m;
    int e;
};

// The high word of a double lies in [2^-64, 2^64): what the functions below take.
__device__ __forceinline__ bool fix_range(double x) { return (uint32_t)__double2hiint(x) - 0x3bf00000u < 0x08000000u; }

// x > 0 (normal): m in [2^63, 2^64).
__device__ __forceinline__ Fix64 fix_of(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return {(b << 11) | 0x8000000000000000ull, (int)(b >> 52) - 1086};
}

// |x| of any normal x.
__device__ __forceinline__ Fix64 fix_abs(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return {(b << 11) | 0x8000000000000000ull, ((int)(b >> 52) & 0x7ff) - 1086};
}

// High 64 bits of a * b, short by less than 3 units (the low x low product and the
// cross terms' fractions are dropped).
__device__ __forceinline__ uint64_t mul_hi(uint64_t a, uint64_t b) {
    const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
    return (uint64_t)ah * bh + (((uint64_t)ah * bl) >> 32) + (((uint64_t)al * bh) >> 32);
}
__device__ __forceinline__ Fix64 operator*(Fix64 a, Fix64 b) { return {mul_hi(a.m, b.m), a.e + b.e + 64}; }

__device__ __forceinline__ Fix64 fix_norm(Fix64 a) {
    const int z = __clzll((long long)(a.m | 1ull));
    return {a.m << z, a.e - z};
}

// The bits of the double nearest to m 2^(biased - 1086) for an exponent field that no normal
// double has: infinity, or a subnormal (ties away from zero) or zero.
__device__ __forceinline__ uint64_t fix_ends(uint64_t m, int biased) {
    if (biased > 0) return 0x7ff0000000000000ull;
    const int s = min(12 - biased, 65);
    return s > 64 ? 0ull : ((m >> (s - 1)) >> 1) + ((m >> (s - 1)) & 1ull);
}

// The double nearest to m * 2^e (ties away from zero).  kEnds false, for results that are
// below 2^1024 by the ranges of what they are formed from: 0 below 2^-1022.
template <bool kEnds = true>
__device__ __forceinline__ double fix_double(Fix64 a) {
    a = fix_norm(a);
    const int biased = a.e + 1086;
    const uint64_t r = (a.m >> 11) + ((a.m >> 10) & 1ull);   // the implicit bit adds 1 to the exponent field
    uint64_t b = ((uint64_t)(uint32_t)(biased - 1) << 52) + r;
    if (kEnds && (uint32_t)(biased - 1) >= 2046u) b = fix_ends(a.m, biased);
    return ((!kEnds && biased <= 0) || (long long)a.m >= 0) ? 0. : __longlong_as_double((long long)b);
}

// The double nearest to a * x * (-1)^negative for a with its top bit set (or 0) and a normal
// x (or 0); kEnds as above.
template <bool kEnds = true>
__device__ __forceinline__ double fix_scale(Fix64 a, double x, bool negative = false) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    uint64_t m = mul_hi(a.m, (b << 11) | 0x8000000000000000ull);   // [2^62, 2^64)
    int biased = a.e + ((int)(b >> 52) & 0x7ff) + 64;
    if ((long long)m >= 0) {
        m <<= 1;
        biased--;
    }
    const uint64_t r = (m >> 11) + ((m >> 10) & 1ull);
    const uint64_t sign = ((b >> 32) & 0x80000000ull) ^ (negative ? 0x80000000ull : 0ull);
    uint64_t v = ((uint64_t)(uint32_t)(biased - 1) << 52) + r;
    if (kEnds && (uint32_t)(biased - 1) >= 2046u) v = fix_ends(m, biased);
    const bool zero = (!kEnds && biased <= 0) || !flag_nonzero(x) || (kEnds && (long long)m >= 0);
    return zero ? 0. : __longlong_as_double((long long)((sign << 32) + v));
}

// 2^114 / M for M in [2^52, 2^53): (2^61, 2^62], error below 2^5 units.
// One third-order Newton step y (1 + e + e^2), e = 1 - M y, from the FP32
// reciprocal of the leading 24 bits (|e| < 2^-21): M y agrees with 2^76 in its
// upper bits, so e is the low 64 bits of the integer product, exactly.
__device__ __forceinline__ uint64_t recip_mant(uint64_t M) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__int_as_float(0x3f800000 | ((int)(M >> 29) & 0x7fffff))));
    r = fmaxf(fminf(r, 0.99999994f), 0.5f);   // [1/2, 1): 24 mantissa bits
    const uint32_t R = ((uint32_t)__float_as_int(r) & 0x7fffffu) | 0x800000u;   // r 2^24
    const long long e = -(long long)(M * (uint64_t)R);                         // e 2^76
    const long long t = (long long)(int)(e >> 32) * (long long)R + (long long)(((uint64_t)(uint32_t)e * R) >> 32);
    const int es = (int)(e >> 39);                                              // e 2^37
    return ((uint64_t)R << 38) + (uint64_t)(t >> 6) + (((uint64_t)R * (uint32_t)(es * es)) >> 36);
}
// 1 / x for x > 0 (normal).
__device__ __forceinline__ Fix64 fix_recip(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    return {recip_mant((b & 0xfffffffffffffull) | 0x10000000000000ull), 961 - (int)(b >> 52)};
}
__device__ __forceinline__ Fix64 fix_recip(float x) {
    const uint32_t b = (uint32_t)__float_as_int(x);
    return {recip_mant((uint64_t)((b & 0x7fffffu) | 0x800000u) << 29), 65 - (int)(b >> 23)};
}
// The double 1 / x, correctly rounded (top bit set): the nearest 53-bit integer
// by the sign of its exact remainder.
__device__ __forceinline__ Fix64 fix_recip_rn(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const uint64_t M = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    uint64_t y = (recip_mant(M) + 256) >> 9;           // 2^105 / M, within 1
    const long long rem = -(long long)(M * y);          // 2^105 - M y
    y += 2 * rem > (long long)M ? 1 : 2 * rem < -(long long)M ? -1 : 0;
    return fix_norm({y << 10, 960 - (int)(b >> 52)});
}

// The double a * x for a double a as its mantissa and a positive normal float x,
// round to nearest even, with its top bit set or (rounded up to a power of two) clear.
__device__ __forceinline__ Fix64 fix_mul_rn(Fix64 a, float x) {
    const uint32_t xb = (uint32_t)__float_as_int(x), xm = (xb << 8) | 0x80000000u;
    const uint64_t lo = (uint64_t)xm * (uint32_t)a.m;
    uint64_t p = (uint64_t)xm * (uint32_t)(a.m >> 32) + (lo >> 32);
    uint32_t rest = (uint32_t)lo;
    int e = a.e + (int)(xb >> 23) - 126;
    if ((long long)p >= 0) {
        p = (p << 1) | (rest >> 31);
        rest <<= 1;
        e--;
    }
    const uint64_t r = (p >> 11) + (((p & 0x7ff) + 0x3ff + (rest || ((p >> 11) & 1))) >> 11);
    return {r << 10, e + 1};
}

// (float)x, round to nearest even, for x whose float is positive and normal.
__device__ __forceinline__ float float_of_normal(double x) {
    uint64_t b = (uint64_t)__double_as_longlong(x);
    b += 0xfffffffull + ((b >> 29) & 1ull);
    return __int_as_float((int)((uint32_t)(b >> 29) - 0xc0000000u));
}

// Any x truncated to a float, for bounds that allow for the error: zero below
// the normal floats, infinity (also for NaN) from 2^127 on.
__device__ __forceinline__ float float_trunc(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const uint32_t hi = (uint32_t)(b >> 32), ex = hi & 0x7fffffffu;
    const uint32_t f = ((uint32_t)(b >> 29) - 0xc0000000u) & 0x7fffffffu;
    const uint32_t g = ex < 0x38100000u ? 0u : ex >= 0x47e00000u ? 0x7f800000u : f;
    return __int_as_float((int)((hi & 0x80000000u) | g));
}

}  // namespace sphfem
