/*
 * FP64 conversions and a division by a constant in integer arithmetic.
 *
 * FP64 instructions, conversions among them, share one pipe of 1.7
 * lane-operations per clock and SM; integer instructions run at 64 and
 * more.  Each function returns exactly what the operator returns; rare
 * operands (subnormal, infinite, NaN, rounding in doubt) take the operator
 * itself.
 */
#pragma once
#include <cuda_runtime.h>

/* (float)x, to nearest even */
__device__ __forceinline__ float f64_to_f32(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned e = (unsigned)(b >> 52) & 0x7ff;
    if (e - 897u < 253u) {   /* normal in FP32, and not rounded up to infinity */
        const unsigned long long r = b + 0x0fffffffull + ((b >> 29) & 1ull);   /* half an ulp, ties to even */
        return __int_as_float((int)((((unsigned)(r >> 29) - (896u << 23)) & 0x7fffffffu) | ((unsigned)(b >> 32) & 0x80000000u)));
    }
    if ((b << 1) == 0ull) return __int_as_float((int)(b >> 32));
    return (float)x;
}
/* (double)x */
__device__ __forceinline__ double f32_to_f64(float x) {
    const unsigned b = (unsigned)__float_as_int(x), e = (b >> 23) & 0xff;
    if (e - 1u < 254u) return __hiloint2double((int)((b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7fffffu) >> 3)), (int)(b << 29));
    if ((b << 1) == 0u) return __hiloint2double((int)b, 0);
    return (double)x;
}
/* (double)v */
__device__ __forceinline__ double i64_to_f64(long long v) {
    const unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
    if (a == 0ull) return 0.0;
    if (a >> 53) return (double)v;
    const int lz = __clzll((long long)a);
    const unsigned long long m = (a << lz) >> 11;   /* 53 bits, the first one set */
    const unsigned long long b = ((unsigned long long)(1085 - lz) << 52) + m;   /* the set bit adds 1 to the exponent */
    return __longlong_as_double((long long)(v < 0 ? b | (1ull << 63) : b));
}

/* Division by a positive normal constant d.  With ma, md the 53-bit
 * mantissas, the upper half of ma 2^11 * floor(2^116 / md) is
 * floor(ma 2^63 / md) less at most 3: ten or eleven bits more than the
 * quotient's 53.  It rounds as the exact quotient does unless those bits
 * are within 3 below or at a half, where the division decides.           */
struct DivBy {
    double d;
    unsigned long long inv;   /* floor(2^116 / md), at most 2^64 - 1 */
    int e;                    /* exponent field of d */
};
inline DivBy div_by(double d) {
    DivBy q;
    unsigned long long b;
    static_assert(sizeof b == sizeof d, "");
    __builtin_memcpy(&b, &d, sizeof b);
    const unsigned long long md = (b & 0xfffffffffffffull) | (1ull << 52);
    const unsigned __int128 inv = ((unsigned __int128)1 << 116) / md;
    q.d = d;
    q.inv = inv >> 64 ? ~0ull : (unsigned long long)inv;
    q.e = (int)(b >> 52);
    if (q.e < 1 || q.e > 2046) q.e = -8192;   /* not positive and normal: no quotient is in range below */
    return q;
}
__device__ __forceinline__ double div_const(double x, const DivBy& D) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    const unsigned long long m = (b << 11) | (1ull << 63);
    const unsigned long long q = __umul64hi(m, D.inv);
    const int up = (int)(q >> 63);   /* 1: quotient of mantissas in [1, 2), else in (1/2, 1) */
    const int e = ex - D.e + 1022 + up;
    const unsigned drop = 10u + up, half = 512u << up, low = (unsigned)q & (2u * half - 1u);
    if ((unsigned)(ex - 1) < 2046u && (unsigned)(e - 1) < 2045u && low - (half - 3u) > 3u) {
        const unsigned long long r = (q >> drop) + (low > half ? 1ull : 0ull);   /* 2^52 .. 2^53 */
        return __longlong_as_double((long long)((((unsigned long long)(e - 1)) << 52) + r) | (long long)(b & (1ull << 63)));
    }
    if ((b << 1) == 0ull) return x;
    return x / D.d;
}
