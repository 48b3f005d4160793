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

__device__ __forceinline__ bool nan64(double x) {
    return (bits64(x) & kMag64) > 0x7ff0000000000000ull;
}
// x < y also where x may be NaN (then false)
__device__ __forceinline__ bool lt64_nan(double x, double y) { return lt64(x, y) && !nan64(x); }
// x > y also where x may be NaN (then false)
__device__ __forceinline__ bool gt64_nan(double x, double y) { return lt64(y, x) && !nan64(x); }
// x <= y also where either may be NaN (then false)
__device__ __forceinline__ bool le64_nan(double x, double y) {
    return !lt64(y, x) && !nan64(x) && !nan64(y);
}
// x > 0 ? x : 0 (0 for a NaN)
__device__ __forceinline__ double above_zero(double x) {
    return bits64(x) - 1 < 0x7ff0000000000000ull ? x : 0.0;
}
// neither is an infinity or NaN
__device__ __forceinline__ bool finite64(double x, double y) {
    return max(hi32(x) & 0x7fffffffu, hi32(y) & 0x7fffffffu) < 0x7ff00000u;
}

// The larger and smaller of two numbers, the second on ties (x > y ? x : y and
// x < y ? x : y, as src/anuga_HMPP/util_ext.h:45-59).
__device__ __forceinline__ double imax(double x, double y) { return lt64(y, x) ? x : y; }
__device__ __forceinline__ double imin(double x, double y) { return lt64(x, y) ? x : y; }
// The smaller where either may be NaN (then the second).
__device__ __forceinline__ double imin_nan(double x, double y) {
    return lt64(x, y) && !nan64(x) && !nan64(y) ? x : y;
}

// 0.5 * x on the integer pipe where the halved number is normal (or x zero)
static __device__ __noinline__ double half_any(double x) { return 0.5 * x; }
__device__ __forceinline__ double half_of(double x) {
    const unsigned h = hi32(x);
    const bool zero = (bits64(x) & kMag64) == 0;
    if (!zero && (h & 0x7ff00000u) - 0x00200000u >= 0x7fd00000u) return half_any(x);
    return __hiloint2double((int)(zero ? h : h - 0x00100000u), __double2loint(x));
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
// B in [2^52, 2^53), A in [B, 2B), b = B / 2^52.  The reciprocal of b's leading
// 24 bits is off by at most 2^-23 / b^2 above (truncation) and 2^-23 either way
// (rcp.approx); scaled by 1 - 2^-21, r never exceeds 1/b and is short of it by a
// factor of at most 1 - (4.5 + b) 2^-23.  The two errors are not largest
// together (the first at b = 1, the second at b = 2), which is what keeps R2
// within the 56 bits that bits23<33> takes:
//   q1 = floor(A r 2^21):   A's 24 bits, a product's rounding and the floor on
//                           top: short by less than (6 + b) / 2 + 1
//                           -> R1 = 2^21 A - q1 B in [0, 5B)
//   q2 = floor(R1 r 2^20):  R1's bits from 2^33 cut up to 2 / b: short by less
//                           than (4 + b / 2) (5 + b) / 8 + 2 / b + 1 <= 6.375
//                           -> R2 in [0, 6.375 B), below 2^55.7
//   q3 = floor(R2 r 2^11):  short by < 1.02 -> R3 in [0, 1.02 B)
// N = 2^31 q1 + 2^11 q2 + q3 and R3 = 2^52 A - N B decide the rounding.
//
// Straight-line code, so that several run interleaved (a warp alone on an SM
// waits out the latency of every instruction of a single one): fine is
// cleared for operands that div_any has to take.
__device__ __forceinline__ double div_digits(double a, double b, bool &fine) {
    const unsigned ha = hi32(a), hb = hi32(b);
    const int ea = (int)((ha >> 20) & 0x7ffu), eb = (int)((hb >> 20) & 0x7ffu);
    const unsigned sign = (ha ^ hb) & 0x80000000u;
    int e = ea - eb + 1022;
    const unsigned la = (unsigned)__double2loint(a), lb = (unsigned)__double2loint(b);
    const bool zero = ((ha << 1) | la) == 0u;
    fine = (unsigned)(eb - 1) < 2046u &&
           (zero || ((unsigned)(ea - 1) < 2046u && (unsigned)(e - 1) < 2043u));
    const unsigned mah = (ha & 0xfffffu) | 0x100000u, mbh = (hb & 0xfffffu) | 0x100000u;
    u64 A = ((u64)mah << 32) | la;
    const u64 B = ((u64)mbh << 32) | lb;
    const float r = rcp_est(lead(mbh, lb)) * 0.99999952316284f;  // 1 - 2^-21
    float af = lead(mah, la);
    const bool small = A < B;
    A = small ? A + A : A;
    af = small ? af + af : af;
    e = small ? e - 1 : e;
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
    N += (u64)((unsigned)e << 20) << 32;
    return from64((zero ? 0ull : N) | ((u64)sign << 32));
}

// Two and three quotients side by side, out of line: the step kernels take
// 13 to 25 of them, and with each in place a kernel was 35 kB of code that a
// small mesh's one warp per SM fetched once per launch (25 us for 2,116
// triangles' distribute).
struct Two {
    double a, b;
};
struct Three {
    double a, b, c;
};
static __device__ __noinline__ Two div2(double a0, double b0, double a1, double b1) {
    bool f0, f1;
    Two q = {div_digits(a0, b0, f0), div_digits(a1, b1, f1)};
    if (!(f0 && f1)) {
        if (!f0) q.a = div_any(a0, b0);
        if (!f1) q.b = div_any(a1, b1);
    }
    return q;
}
static __device__ __noinline__ Three div3(double a0, double b0, double a1, double b1, double a2,
                                          double b2) {
    bool f0, f1, f2;
    Three q = {div_digits(a0, b0, f0), div_digits(a1, b1, f1), div_digits(a2, b2, f2)};
    if (!(f0 && f1 && f2)) {
        if (!f0) q.a = div_any(a0, b0);
        if (!f1) q.b = div_any(a1, b1);
        if (!f2) q.c = div_any(a2, b2);
    }
    return q;
}
static __device__ __noinline__ double fdiv64(double a, double b) {
    bool fine;
    const double q = div_digits(a, b, fine);
    return fine ? q : div_any(a, b);
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
__device__ __forceinline__ double sqrt_digits(double x, bool &fine) {
    const unsigned hx = hi32(x), lx = (unsigned)__double2loint(x);
    const bool zero = ((hx << 1) | lx) == 0u;
    fine = hx - 0x00100000u < 0x7fe00000u || zero;  // normal and positive, or a zero
    const unsigned ex = hx >> 20;
    const unsigned mh = (hx & 0xfffffu) | 0x100000u;
    u64 X = ((u64)mh << 32) | lx;
    float xf = lead(mh, lx);
    const bool odd = !(ex & 1u);  // the unbiased exponent
    X = odd ? X + X : X;
    xf = odd ? xf + xf : xf;
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
    N += (u64)(e << 20) << 32;
    return zero ? x : from64(N);
}
static __device__ __noinline__ Two sqrt2(double x0, double x1) {
    bool f0, f1;
    Two r = {sqrt_digits(x0, f0), sqrt_digits(x1, f1)};
    if (!(f0 && f1)) {
        if (!f0) r.a = sqrt_any(x0);
        if (!f1) r.b = sqrt_any(x1);
    }
    return r;
}
__device__ __forceinline__ double fsqrt64(double x) {
    bool fine;
    const double r = sqrt_digits(x, fine);
    return fine ? r : sqrt_any(x);
}

// ---- h^(7/3) ---------------------------------------------------------------

static __device__ __noinline__ double pow73_any(double h) { return pow(h, 7.0 / 3); }

// h to the FP64 number nearest 7/3, within 0.52 ulp (pow: within 1): h^2 and
// the cube root of h each as a pair, the root from an FP32 estimate c of 24
// bits by two terms of the binomial series, c (1 + x/3 - x^2/9), x = h/c^3 - 1
// of 2^-20, h / c^3 a quotient of the integer pipe; the exponent's own
// rounding, 1.48e-16, by its first-order term.  14 FP64 instructions; pow
// executes about 80.
__device__ __forceinline__ double pow_seven_thirds(double h) {
    const unsigned hh = hi32(h);
    if (hh - 0x3c300000u >= 0x07900000u) return pow73_any(h);  // outside [2^-60, 2^61)
    const float hf = __uint_as_float(__funnelshift_l((unsigned)__double2loint(h),
                                                     hh - (896u << 20), 3));
    float lg, cf;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(hf));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(cf) : "f"(lg * 0.33333333f));
    const auto widen32 = [](float v) {  // normal v
        const unsigned u = __float_as_uint(v);
        return __hiloint2double((int)((((u & 0x7fffffffu) >> 3) + (896u << 20)) |
                                      (u & 0x80000000u)),
                                (int)(u << 29));
    };
    const double c = widen32(cf);
    const double c2 = c * c;                   // exact: 48 bits
    const double r = fma(-c2, c, h);           // h - c^3
    const double x = fdiv64(r, c2 * c);
    const double u = x * (1.0 / 3);
    const double cl = c * fma(-u, u, u);       // the root is c + cl
    const double p = h * h, pl = fma(h, h, -p);
    const double q = p * c;
    double s = fma(p, c, -q);
    s = fma(p, cl, s);
    s = fma(pl, c, s);
    // 1.4802973661668753e-16 ln h = 1.0260639499e-16 log2 h (zero widens to 2^-127)
    s = fma(q, widen32(lg * 1.0260639e-16f), s);
    return q + s;
}

}  // namespace swgpu
