// 64-bit fixed-point arithmetic on the integer pipe for the plain path.
//
// On GB300 an FP64 instruction occupies its sub-partition for 64 cycles (measured), a 32 x 32 + 64-bit
// multiply-add (mad.wide) for 4 and other integer instructions for 2: a term of a dot product takes
// three mad.wide (hi hi, hi lo, lo hi) instead of one FP64 FMA, and an exponential about 50 integer
// instructions instead of 9 FP64 ones. The integer and FP64 pipes run side by side.
//
// Accuracy: logarithms are kept to 2^-51 absolute, which is the relative error of their exponential;
// an FP64 evaluation of the exponent rounds at 2^-53 of its magnitude (about 2^-47 at 40).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_math.cuh"
#include "tables_fixed.h"

namespace cbg {

__device__ __forceinline__ const FixMath& fmath() { return *reinterpret_cast<const FixMath*>(cb_dsmem + kMathBytes); }

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long mul_wide_u(unsigned a, unsigned b) {
    unsigned long long d;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
}

// Words of a fixed-point integer (|v| < 2^60): v = hi 2^LO + lo, lo balanced.
template <int LO = kLo>
__device__ __forceinline__ Word2 split_word(long long v) {
    Word2 w;
    w.hi = (int)((v + (1ll << (LO - 1))) >> LO);
    w.lo = (int)(v - ((long long)w.hi << LO));
    return w;
}

// One term of a dot product: hi words into s1, cross products into s2 (2^-29 of s1's unit); lo lo dropped.
__device__ __forceinline__ void dot_term(const Word2& a, const Word2& b, long long& s1, long long& s2) {
    s1 = mad_wide(a.hi, b.hi, s1);
    s2 = mad_wide(a.hi, b.lo, s2);
    s2 = mad_wide(a.lo, b.hi, s2);
}
__device__ __forceinline__ long long dot_value(long long s1, long long s2) {
    return s1 + ((s2 + (1ll << (kLo - 1))) >> kLo);
}

// x 2^q as an integer, rounded to nearest; |x| 2^q < 2^61.
__device__ __forceinline__ long long dbl_to_fix(double x, int q) {
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff) - 1023 + q;  // |x| 2^q in [2^e, 2^(e+1))
    const unsigned long long m = ((unsigned long long)b << 10 | (1ull << 62)) & 0x7ffffffffffffc00ull;
    const long long v = e < -1 ? 0 : (long long)(((m >> (61 - e)) + 1) >> 1);
    return b < 0 ? -v : v;
}

// v 2^-q as a double, rounded to nearest (ties away); any v above -2^63.
__device__ __forceinline__ double fix_to_dbl(long long v, int q) {
    if (v == 0) return 0.0;
    const unsigned long long a = v < 0 ? (unsigned long long)(-v) : (unsigned long long)v;
    const int lz = __clzll((long long)a);
    unsigned long long m = a << lz;                      // [2^63, 2^64)
    const unsigned long long r = m >> 11;                // 53 bits
    const long long bits = ((long long)(63 - lz - q + 1022) << 52) + (long long)r + (long long)((m >> 10) & 1);
    return __longlong_as_double(bits | (v < 0 ? (long long)0x8000000000000000ull : 0ll));
}

// (ah 2^32 + al)(bh 2^32 + bl) / 2^64 to two units: lo lo and the cross products' low words dropped. The
// cross products' high words must fit 32 bits together.
__device__ __forceinline__ unsigned long long mul_hi3(unsigned ah, unsigned al, unsigned bh, unsigned bl) {
    unsigned long long d;
    asm("{\n .reg .u32 s, z;\n .reg .u64 c;\n mul.hi.u32 s, %1, %4;\n mad.hi.u32 s, %2, %3, s;\n mov.u32 z, 0;\n"
        " mov.b64 c, {s, z};\n mad.wide.u32 %0, %1, %3, c;\n}"
        : "=l"(d) : "r"(ah), "r"(al), "r"(bh), "r"(bl));
    return d;
}

// 2^(y 2^-51) for -1021 <= y 2^-51 < 1023: 1024 table points, u the position between two of them, and
// 2^(u/1024) - 1 = c u (1 + c u/2 + (c u)^2/6 + (c u)^3/24), c = ln2 / 1024 (next term below 2^-59). The words of the
// factor in brackets leave up to 1.3 2^-52 (0.22 rms): two coefficients are one up, which centres the truncations (2.5 and 0.53 without).
__device__ __forceinline__ double exp2_core(long long y) {
    const unsigned yh = (unsigned)(y >> 32), yl = (unsigned)y;
    const unsigned long long t = fmath().exp2t[(yh >> 9) & (kExpTable - 1)];  // Q62
    const unsigned u = __funnelshift_l(yl, yh, 23), ul = yl << 23;            // u, Q32, and its next 9 bits
    unsigned h = __umulhi(u, 114u);                                           // Q43
    h = __umulhi(u, 671723u + h);
    h = __umulhi(u, 2977044473u + h);
    const unsigned long long w = mul_hi3(u, ul, 0x0B17217Fu, 0x7D1CF79Bu);    // u ln2, Q60
    const unsigned long long q = w + (mul_wide_u((unsigned)(w >> 28), h) >> 15);
    const unsigned long long tq = mul_hi3((unsigned)(q >> 32), (unsigned)q, (unsigned)(t >> 32), (unsigned)t);
    const unsigned long long m = t + (tq >> 6);
    return __longlong_as_double(((long long)(((int)yh >> 19) + 1022) << 52) + (long long)((m + 512) >> 10));
}
static __device__ __noinline__ double exp2_slow(double y) { return exp2(y); }
static __device__ __noinline__ double exp2_slow_fix(long long y) {
    if (y < -(1076ll << kYq)) return 0.0;  // (no FP64 instructions: at low temperatures many)
    return exp2((double)y * 0x1p-51);
}
__device__ __forceinline__ double exp2_fix(long long y) {
    // -1021 <= y < 1023 by the high word
    if ((unsigned)((int)(y >> 32) + (1021 << 19)) >= (2044u << 19)) return exp2_slow_fix(y);
    return exp2_core(y);
}
// min(f32::MAX, 2^y) (reaction.rs:138), or of the constant that y stands for (kConstRate); from 128 - 2^-18 on out of line.
static __device__ __noinline__ double rate_slow(long long y) {
    if (y >= kConstRateMin) return min_pos(kF32Max, __longlong_as_double(y - kConstRate));
    if (y >= (128ll << kYq)) return kF32Max;
    if (y < -(1076ll << kYq)) return 0.0;
    return min_pos(kF32Max, exp2((double)y * 0x1p-51));
}
__device__ __forceinline__ double rate_fix(long long y) {
    if ((unsigned)((int)(y >> 32) + (1021 << 19)) >= (1149u << 19) - 2u) return rate_slow(y);
    return exp2_core(y);
}
// 2^y of a double.
__device__ __forceinline__ double exp2_dbl(double y) {
    if ((__double2hiint(y) & 0x7fffffff) >= 0x408fe800) return exp2_slow(y);  // |y| >= 1021, inf or NaN
    return exp2_core(dbl_to_fix(y, kYq));
}

// log2 of a positive normal x: exponent and a 62-bit fraction. x = 2^e F, F rc = 1 + u exactly (rc a 12-bit
// reciprocal of the table point), log2 F = -log2 rc + log2(e) (u - u^2/2 + u^2 (u/3 - u^2/4 + u^3/5))
// (|u| <= 1.3 2^-10, next term below 2^-60).
__device__ __forceinline__ long long log2_frac(double x, int& e) {
    const long long b = __double_as_longlong(x);
    e = (int)(b >> 52) - 1023;
    const unsigned long long F = ((unsigned long long)b & 0xfffffffffffffull) | (1ull << 52);
    const int j = (int)((b >> 43) & 511);
    const long long u = (long long)(F * fmath().rc[j]);  // Q64, modulo 1
    const long long u2 = __mul64hi(u, u);                // Q64
    const int v = (int)(u >> 24), w = (int)(u2 >> 14);   // Q40, Q50
    int p = 429496730;                                   // 1/5, Q31
    p = -536870912 + (__mulhi(v, p) >> 8);
    p = 715827883 + (__mulhi(v, p) >> 8);
    const int s = __mulhi(v, p);                                      // Q39
    const long long l = u - (u2 >> 1) + (mad_wide(w, s, 0) >> 25);    // ln(1 + u), Q64
    return fmath().log2c[j] + ((l + __mul64hi(l, 0x71547652B82FE177ll)) >> 2);  // times log2(e), Q62
}
// log2(x), Q51.
__device__ __forceinline__ long long log2_fix(double x) {
    int e;
    const long long f = log2_frac(x, e);
    return ((long long)e << kYq) + ((f + (1ll << 10)) >> 11);
}
static __device__ __noinline__ double log2_slow(double x) { return log2(x); }
// log2(x) as a double, any x.
__device__ __forceinline__ double log2_dbl(double x) {
    const int hi = __double2hiint(x);
    if (hi < 0x00100000 || hi >= 0x7ff00000) return log2_slow(x);  // <= 0, subnormal, inf or NaN
    return fix_to_dbl(log2_fix(x), kYq);
}


// 1 / (d 2^-60 2^sp) for 2^54 < d < 2^61, as a double; bias = PolyX::rcp_bias. A 24-bit estimate R0 2^-84 of 1/d,
// its residual e = 1 - d R0 2^-84 exactly (modulo 2^64), and R0 (1 + e + e^2): e^3 is below 2^-60.
__device__ __forceinline__ double rcp_fixed(long long d, int bias) {
    const float f = __uint2float_rn((unsigned)(d >> 30));
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(f));
    const unsigned R0 = __float2uint_rn(r0 * 0x1p54f);
    const long long e = -(long long)((unsigned long long)d * R0);  // Q84
    const int eh = (int)(e >> 32);                                 // Q52
    const long long s = e + (mad_wide(eh, eh, 0) >> 20);
    const long long corr = mad_wide((int)R0, (int)(s >> 32), 0) + __umulhi(R0, (unsigned)s);  // R0 s, Q52
    const unsigned long long R = ((unsigned long long)R0 << 32) + (unsigned long long)(corr >> 20);
    const int lz = __clz((int)(R >> 32));
    const unsigned hi = __funnelshift_l((unsigned)R, (unsigned)(R >> 32), lz), lo = (unsigned)R << lz;
    const unsigned long long m = ((unsigned long long)hi << 32) | lo;
    return __longlong_as_double(((long long)(bias - lz) << 52) + (long long)(m >> 11) + (long long)((m >> 10) & 1));
}

}  // namespace cbg
