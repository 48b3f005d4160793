// swgpu_soft64.cuh -- FP64 division, square root and comparisons on the
// integer and FP32 pipes, with the results of IEEE arithmetic bit for bit.
//
// GB300 issues two FP64 thread instructions per SM and clock, against 128 of
// the other pipes: an FP64 instruction costs a warp 16 SM clocks, a division
// or square root of about ten of them 160, and a comparison as much as an
// addition.  The quotient and root below are 65-70 integer and FP32
// instructions (about 30 SM clocks beside an FP64 pipe that they leave free)
// and their result is the correctly rounded one, so it does not depend on
// which of the two computed it.
//
// Method: digit recurrences of very high radix (21, 20 and 11 bits), each
// digit an underestimate from an FP32 reciprocal (or reciprocal root) of the
// leading bits, each remainder exact in 64-bit integers modulo 2^64; the last
// remainder decides the rounding.  A quotient or root of two normal numbers
// is never half way between two FP64 numbers, so no tie rule is needed.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace swgpu {

typedef unsigned long long u64;
typedef long long i64;

__device__ __forceinline__ u64 bits64(double x) { return (u64)__double_as_longlong(x); }
__device__ __forceinline__ double from64(u64 b) { return __longlong_as_double((i64)b); }
__device__ __forceinline__ unsigned hi32(double x) { return (unsigned)__double2hiint(x); }

// ---- comparisons ----------------------------------------------------------
// IEEE results for operands that are not NaN (either zero equals the other).

constexpr u64 kMag64 = 0x7fffffffffffffffull;

// |x| < |y|: also x < y where neither is below zero (a zero of either sign
// allowed)
__device__ __forceinline__ bool mag_lt(double x, double y) {
    return (bits64(x) & kMag64) < (bits64(y) & kMag64);
}
// x < c for a c above zero
__device__ __forceinline__ bool lt_pos(double x, double c) {
    return (i64)bits64(x) < (i64)bits64(c);
}
__device__ __forceinline__ bool gt_zero(double x) { return (i64)bits64(x) > 0; }
__device__ __forceinline__ bool lt_zero(double x) { return bits64(x) > 0x8000000000000000ull; }
__device__ __forceinline__ bool ge_zero(double x) { return !lt_zero(x); }
// sign and magnitude as a two's complement number (both zeros are 0)
__device__ __forceinline__ i64 order64(double x) {
    const i64 b = (i64)bits64(x), s = b >> 63;
    return ((b & (i64)kMag64) ^ s) - s;
}
__device__ __forceinline__ bool lt64(double x, double y) { return order64(x) < order64(y); }

// x < y also where x may be NaN (then false)
__device__ __forceinline__ bool lt64_nan(double x, double y) {
    return lt64(x, y) && (bits64(x) & kMag64) <= 0x7ff0000000000000ull;
}

// The larger and smaller of two, the second on ties (x > y ? x : y and
// x < y ? x : y, as src/anuga_HMPP/util_ext.h:45-59).
__device__ __forceinline__ double imax(double x, double y) { return lt64(y, x) ? x : y; }
__device__ __forceinline__ double imin(double x, double y) { return lt64(x, y) ? x : y; }

// 0.5 * x on the integer pipe where the halved number is normal (or x zero)
__device__ __forceinline__ double half_of(double x) {
    const unsigned h = hi32(x), e = h & 0x7ff00000u;
    if (e - 0x00200000u < 0x7fd00000u)  // exponent 2 .. 2046
        return __hiloint2double((int)(h - 0x00100000u), __double2loint(x));
    if ((bits64(x) & kMag64) == 0) return x;
    return 0.5 * x;
}

// ---- division and square root ---------------------------------------------

// Out of line: operands outside the normal range, and results near its ends.
static __device__ __noinline__ double div_any(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_any(double x) { return sqrt(x); }

__device__ __forceinline__ float rcp_est(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_est(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// floor of 0 <= x < 2^23
__device__ __forceinline__ unsigned floor23(float x) {
    return __float_as_uint(__fadd_rd(x, 8388608.0f)) & 0x7fffffu;
}
// the 23 bits of v from bit `at` up, as a float (v < 2^(at + 23))
template <int at>
__device__ __forceinline__ float bits23(u64 v) {
    return __uint_as_float(0x4b000000u | (unsigned)(v >> at)) - 8388608.0f;
}
// the leading bits of a 53-bit significand m as a float in [1, 2)
__device__ __forceinline__ float lead(unsigned mh, unsigned ml) {
    return __uint_as_float(0x3f800000u | (__funnelshift_l(ml, mh, 3) & 0x7fffffu));
}
__device__ __forceinline__ u64 mul_32x64(unsigned a, u64 b) {
    return (u64)a * (unsigned)b + ((u64)(a * (unsigned)(b >> 32)) << 32);
}

// a / b, correctly rounded.
//
// B in [2^52, 2^53), A in [B, 2B).  Estimates: the reciprocal r of B's leading
// 24 bits is within 2^-23 (truncation) + 2^-23 (rcp.approx) of 1/B; scaled by
// 1 - 2^-21 it never exceeds it, and is below it by at most 2^-20.4.
//   q1 = floor(A r 2^21):   short by < 2^22 2^-20.4 + 3 (A's 24 bits, floor)
//                           -> R1 = 2^21 A - q1 B in [0, 7B)
//   q2 = floor(R1 r 2^20):  R1's 23 bits from 2^33 cut 2^-19 B: short by
//                           < 7 2^20 2^-20.4 + 2 + 1 -> R2 in [0, 9B)
//   q3 = floor(R2 r 2^11):  short by < 1.02 -> R3 in [0, 1.02 B)
// N = 2^31 q1 + 2^11 q2 + q3 and R3 = 2^52 A - N B decide the rounding.
__device__ __forceinline__ double fdiv64(double a, double b) {
    const unsigned ha = hi32(a), hb = hi32(b);
    const int ea = (int)((ha >> 20) & 0x7ffu), eb = (int)((hb >> 20) & 0x7ffu);
    const unsigned sign = (ha ^ hb) & 0x80000000u;
    int e = ea - eb + 1023;
    const unsigned la = (unsigned)__double2loint(a), lb = (unsigned)__double2loint(b);
    const bool b_normal = (unsigned)(eb - 1) < 2046u;
    if (!(b_normal && (unsigned)(ea - 1) < 2046u && (unsigned)(e - 2) < 2043u)) {
        if (b_normal && (((ha << 1) | la) == 0u)) return __hiloint2double((int)sign, 0);
        return div_any(a, b);
    }
    const unsigned mah = (ha & 0xfffffu) | 0x100000u, mbh = (hb & 0xfffffu) | 0x100000u;
    u64 A = ((u64)mah << 32) | la;
    const u64 B = ((u64)mbh << 32) | lb;
    const float r = rcp_est(lead(mbh, lb)) * 0.99999952316284f;  // 1 - 2^-21
    float af = lead(mah, la);
    if (A < B) {
        A += A;
        af += af;
        e -= 1;
    }
    const unsigned q1 = floor23((af * r) * 2097152.0f);
    const u64 R1 = (A << 21) - mul_32x64(q1, B);
    // R / 2^33 times r / 2^52 in units of the next digit: 2^33 2^20 / 2^52
    const unsigned q2 = floor23(bits23<33>(R1) * (r * 2.0f));
    const u64 R2 = (R1 << 20) - mul_32x64(q2, B);
    const unsigned q3 = floor23(bits23<33>(R2) * (r * 0.00390625f));
    const u64 R3 = (R2 << 11) - mul_32x64(q3, B);
    u64 N = ((u64)q1 << 31) + ((u64)q2 << 11) + q3;
    const u64 t = R3 + R3;
    N += t > B ? 1u : 0u;
    N += t > B + B + B ? 1u : 0u;
    // N in [2^52, 2^53]: its leading bit adds one to the exponent field
    return from64(N + ((u64)(((unsigned)(e - 1) << 20) | sign) << 32));
}

// sqrt(x), correctly rounded.
//
// X in [2^52, 2^54) with an even exponent, S = sqrt(2^52 X) in [2^52, 2^53).
// The estimate y of 1/sqrt(X / 2^52) from 24 leading bits is within 2^-22,
// scaled by 1 - 2^-21 it does not exceed it.
//   s1 = floor(x y 2^21), R1 = X - 2^10 s1^2 < 2^36
//   s2 = floor(t - 2^-42 t^2), t = 2^9 R1 / s1 (the second term: s2^2's own
//        part of the remainder), R2 = 2^30 R1 - 2^21 s1 s2 - s2^2 < 2^48
//   s3 = floor(R2 / (2^10 s1)), R3 = 2^22 R2 - 2^32 s1 s3 - 2^12 s2 s3 - s3^2
// N = 2^31 s1 + 2^11 s2 + s3 and R3 = 2^52 X - N^2 decide the rounding (s3,
// which leaves s2 out of its divisor, may exceed the root by up to 0.03: R3
// is then below zero, and above -N / 2, and N stands).
__device__ __forceinline__ double fsqrt64(double x) {
    const unsigned hx = hi32(x), lx = (unsigned)__double2loint(x);
    // normal and positive
    if (hx - 0x00100000u >= 0x7fe00000u) {
        if (((hx << 1) | lx) == 0u) return x;
        return sqrt_any(x);
    }
    const unsigned ex = hx >> 20;
    const unsigned mh = (hx & 0xfffffu) | 0x100000u;
    u64 X = ((u64)mh << 32) | lx;
    float xf = lead(mh, lx);
    if (!(ex & 1u)) {  // the unbiased exponent is odd
        X += X;
        xf += xf;
    }
    const float y = rsqrt_est(xf) * 0.99999952316284f;
    const unsigned s1 = floor23((xf * y) * 2097152.0f);
    const u64 R1 = X - ((u64)s1 * s1 << 10);
    const float est = bits23<13>(R1) * (y + y);  // 1 / s1 = 2^-21 y
    const unsigned s2 = floor23(fmaf(est * est, -2.2737368e-13f, est));  // 2^-42
    const u64 R2 = (R1 << 30) - ((u64)s1 * s2 << 21) - (u64)s2 * s2;
    const unsigned s3 = floor23(bits23<26>(R2) * (y * 0.03125f));
    const u64 R3 = (R2 << 22) - ((u64)s1 * s3 << 32) - ((u64)s2 * s3 << 12) - (u64)s3 * s3;
    u64 N = ((u64)s1 << 31) + ((u64)s2 << 11) + s3;
    const u64 S = N;
    N += (i64)R3 > (i64)S ? 1u : 0u;
    N += (i64)R3 > (i64)(3 * S + 2) ? 1u : 0u;
    // (ex - 1023) / 2 rounded down, plus the bias, less the leading bit's one
    const unsigned e = ((ex + 1023u) >> 1) - 1u;
    return from64(N + ((u64)(e << 20) << 32));
}

}  // namespace swgpu
