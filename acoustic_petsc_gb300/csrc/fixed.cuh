// fixed.cuh -- 64-bit fixed point and significand arithmetic on the integer pipe, for kernels that FP64 issue
// would bound: measured, a warp instruction holds the FP64 pipe for 64 cycles of its scheduler, a 64-bit
// integer addition takes 2, an IMAD.WIDE 4.4 and a 64 x 64 bit product's upper half 17.  The functions are
// host functions too, where they are checked against extended precision.
#pragma once

#include <math.h>
#include <string.h>

namespace hype {
namespace euler {

typedef unsigned long long u64;
typedef long long i64;

__host__ __device__ __forceinline__ u64 umulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
__host__ __device__ __forceinline__ int clz64(u64 x) {  // x != 0
#ifdef __CUDA_ARCH__
    return __clzll((i64)x);
#else
    return __builtin_clzll(x);
#endif
}
__host__ __device__ __forceinline__ i64 bits_of(double x) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(x);
#else
    i64 b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
__host__ __device__ __forceinline__ double from_bits(u64 b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((i64)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}

// A 64-bit integer as h 2^32 + l with a signed l, so that every partial product is a signed 32 x 32 one
// (IMAD.WIDE, with a 64-bit addend for free): 4 of them and 2 shifts an exact 128-bit product, where the
// compiler's own 64 x 64 sequence takes twice the instructions.
struct Split {
    int h, l;
};
__host__ __device__ __forceinline__ Split split(i64 x) {
    const int l = (int)x;
    return Split{(int)(x >> 32) + (int)((unsigned)l >> 31), l};
}
__host__ __device__ __forceinline__ i64 wide(int a, int b, i64 c) { return (i64)a * b + c; }
__host__ __device__ __forceinline__ i64 high(i64 x) { return (i64)(int)(x >> 32); }

// an exact signed 128-bit sum of products; |a.h b.l + a.l b.h| < 2^62 for the operands used here
struct Sum128 {
    u64 hi, lo;
};
__host__ __device__ __forceinline__ Sum128 times128(Split a, Split b) {
    const i64 ll = wide(a.l, b.l, 0);
    const i64 mid = wide(a.l, b.h, wide(a.h, b.l, high(ll)));
    const i64 hh = wide(a.h, b.h, high(mid));
    return Sum128{(u64)hh, ((u64)(unsigned)mid << 32) | (unsigned)ll};
}
__host__ __device__ __forceinline__ Sum128 square128(Split a) {
    const i64 ll = wide(a.l, a.l, 0);
    const i64 mid = wide(2 * a.h, a.l, high(ll));
    const i64 hh = wide(a.h, a.h, high(mid));
    return Sum128{(u64)hh, ((u64)(unsigned)mid << 32) | (unsigned)ll};
}
__host__ __device__ __forceinline__ Sum128 operator+(Sum128 a, Sum128 b) {
#ifdef __CUDA_ARCH__
    Sum128 r;
    asm("add.cc.u64 %0, %2, %4;\n\taddc.u64 %1, %3, %5;" : "=l"(r.lo), "=l"(r.hi) : "l"(a.lo), "l"(a.hi), "l"(b.lo), "l"(b.hi));
    return r;
#else
    const u64 lo = a.lo + b.lo;
    return Sum128{a.hi + b.hi + (lo < a.lo), lo};
#endif
}
__host__ __device__ __forceinline__ Sum128 operator-(Sum128 a, Sum128 b) {
#ifdef __CUDA_ARCH__
    Sum128 r;
    asm("sub.cc.u64 %0, %2, %4;\n\tsubc.u64 %1, %3, %5;" : "=l"(r.lo), "=l"(r.hi) : "l"(a.lo), "l"(a.hi), "l"(b.lo), "l"(b.hi));
    return r;
#else
    return Sum128{a.hi - b.hi - (a.lo < b.lo), a.lo - b.lo};
#endif
}
// x k for a non-negative x and a small k
__host__ __device__ __forceinline__ Sum128 scale128(Sum128 x, unsigned k) {
    const u64 a = (u64)(unsigned)x.lo * k, b = (u64)(unsigned)(x.lo >> 32) * k + (a >> 32);
    return Sum128{x.hi * k + (b >> 32), (b << 32) | (unsigned)a};
}
// x c / 2^64 for a non-negative x
__host__ __device__ __forceinline__ Sum128 part128(Sum128 x, u64 c) {
    const u64 r = x.hi * c, l = umulhi(x.lo, c);
    return Sum128{umulhi(x.hi, c) + (r + l < r), r + l};
}

// x c / 2^64 to within a unit, c below 2^62
__host__ __device__ __forceinline__ i64 scaled(i64 x, Split c) {
    const int h = (int)(x >> 32);
    const i64 mid = (i64)((u64)(unsigned)x * (unsigned)c.h) + wide(h, c.l, 1ll << 31);
    return wide(h, c.h, high(mid));
}
// x w / 2^62, rounded
__host__ __device__ __forceinline__ i64 times62(Split x, Split w) {
    const i64 ll = wide(x.l, w.l, 1ll << 61);
    const i64 mid = wide(x.l, w.h, wide(x.h, w.l, high(ll)));
    const i64 hh = wide(x.h, w.h, high(mid));
    return (hh << 2) | (i64)((unsigned)mid >> 30);
}

// 24 leading bits of 1/m and 1/sqrt(m) in units of 2^-32 from the approximate FP32 instructions: m with 2^31
// for one in [1, 2) and 2^30 for one in [1, 4)
__host__ __device__ __forceinline__ unsigned seed_of(float r) {  // r in [1/2, 1] up to its error
#ifdef __CUDA_ARCH__
    unsigned b = __float_as_uint(r);
#else
    unsigned b;
    memcpy(&b, &r, 4);
#endif
    b = b < 0x3F000000u ? 0x3F000000u : b;
    b = b > 0x3F7FFFFFu ? 0x3F7FFFFFu : b;
    return (b << 8) | 0x80000000u;
}
__host__ __device__ __forceinline__ unsigned rcp_seed(unsigned m) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(((m >> 8) & 0x7FFFFFu) | 0x3F800000u)));
    return seed_of(r);
#else
    return seed_of(1.0f / ((float)(m >> 8) / 8388608.0f));
#endif
}
__host__ __device__ __forceinline__ unsigned rsqrt_seed(unsigned m) {
    // m >= 2^31: [2, 4), exponent 128 and the bits below the leading one; else [1, 2)
#ifdef __CUDA_ARCH__
    const unsigned top = m >> 31;
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float((((m << (1 - top)) >> 8) & 0x7FFFFFu) | (0x3F800000u + (top << 23)))));
    return seed_of(r);
#else
    return seed_of((float)(1.0 / sqrt((double)m / 1073741824.0)));
#endif
}
// 2^127 / m for m in [2^63, 2^64), to within 2^4: with Y the seed and e = 1 - m Y, Y (1 + e + e^2)
__host__ __device__ __forceinline__ u64 recip64(u64 m) {
    const unsigned Y = rcp_seed((unsigned)(m >> 32));
    const u64 q = (u64)(unsigned)(m >> 32) * Y + (((u64)(unsigned)m * Y) >> 32);  // m Y, 2^63 for one
    const i64 e = (i64)((1ull << 63) - q);                                        // at most 2^41
    const int s = (int)(e >> 21);
    const i64 c = e + (wide(s, s, 0) >> 21);
    return ((u64)Y << 32) + (u64)(((c >> 3) * (i64)(Y >> 8)) >> 20) - 6;
}
// 2^31 sqrt(x) for x in [2^62, 2^64): g = x Y, e = 1 - g Y, g (1 + e/2 + 3 e^2/8), 2^62 for one (x = 2^62)
__host__ __device__ __forceinline__ u64 sqrt64(u64 x) {
    const unsigned Y = rsqrt_seed((unsigned)(x >> 32));
    const u64 g = (u64)(unsigned)(x >> 32) * Y + (((u64)(unsigned)x * Y) >> 32);
    const u64 q = (u64)(unsigned)(g >> 32) * Y + (((u64)(unsigned)g * Y) >> 32);
    const i64 e = (i64)((1ull << 62) - q);  // at most 2^41
    const int s = (int)(e >> 20);
    const i64 c = (e >> 1) + ((3 * wide(s, s, 0)) >> 25);
    return g + (u64)(scaled(c << 20, split((i64)(g >> 1))) >> 17);
}

// 2^95 / sqrt(x) for x in [2^62, 2^64): Y (1 + e/2 + 3 e^2/8), e = 1 - x Y^2
__host__ __device__ __forceinline__ u64 rsqrt64(u64 x) {
    const unsigned Y = rsqrt_seed((unsigned)(x >> 32));
    const u64 g = (u64)(unsigned)(x >> 32) * Y + (((u64)(unsigned)x * Y) >> 32);
    const u64 q = (u64)(unsigned)(g >> 32) * Y + (((u64)(unsigned)g * Y) >> 32);
    const i64 e = (i64)((1ull << 62) - q);
    const int s = (int)(e >> 20);
    const i64 c = (e >> 1) + ((3 * wide(s, s, 0)) >> 25);
    return ((u64)Y << 32) + (u64)(((c >> 2) * (i64)(Y >> 8)) >> 20) - 6;
}

// a finite double with biased exponent e <= top as an integer: 2^(52 + SHIFT) stands for 2^(top - 1023)
template <int SHIFT>
__host__ __device__ __forceinline__ i64 to_fixed(i64 b, int top) {
    const int e = (int)(b >> 52) & 0x7FF;
    const u64 m = ((b & 0xFFFFFFFFFFFFFll) | 0x10000000000000ll) << SHIFT;
#ifdef __CUDA_ARCH__
    i64 v;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(top - e));  // shifts of 64 and more, and negative ones, give 0
#else
    const i64 v = (i64)(top - e < 64 ? m >> (top - e) : 0);
#endif
    return b < 0 ? -v : v;
}
// v * 2^(top - 1023 - 58) rounded to the nearest double; the result's exponent is in range by the clamp of
// top.  The conversion instruction is the FP64 pipe's, which the integer form leaves idle.
__host__ __device__ __forceinline__ double from_fixed(i64 v, int top) {
#ifdef __CUDA_ARCH__
    const double d = __ll2double_rn(v);
    return __hiloint2double(__double2hiint(d) + (v ? (top - 1023 - 58) << 20 : 0), __double2loint(d));
#else
    return ldexp((double)v, top - 1023 - 58);
#endif
}
// A positive number m 2^x with the leading bit of m set
struct Norm {
    u64 m;
    int x;
};
__host__ __device__ __forceinline__ Norm norm128(Sum128 J) {  // J != 0
    const bool small = J.hi == 0;
    const u64 hi = small ? J.lo : J.hi, lo = small ? 0 : J.lo;
    const int c = clz64(hi);
    return Norm{(hi << c) | ((lo >> 1) >> (63 - c)), (small ? 0 : 64) - c};
}
// v 2^-s, s of either sign, v 2^-s below 2^64
__host__ __device__ __forceinline__ u64 shift_by(u64 v, int s) {
#ifdef __CUDA_ARCH__
    u64 r;  // shifts of 64 and more give 0
    if (s >= 0) asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    else r = v << -s;
    return r;
#else
    return s >= 64 ? 0 : s >= 0 ? v >> s : v << -s;
#endif
}

// m 2^x, leading bit of m set, rounded to a double
__host__ __device__ __forceinline__ double pack(u64 m, int x) {
    return from_bits(((u64)(x + 63 + 1023 - 1) << 52) + ((m >> 11) + ((m >> 10) & 1)));
}
// from_fixed on the integer pipe, for kernels that FP64 issue bounds
__host__ __device__ __forceinline__ double double_of(i64 v, int top) {
    const u64 s = (u64)(v >> 63), m = ((u64)v ^ s) - s;
    const int c = clz64(m | 1);
    return from_bits((s & 0x8000000000000000ull) | (m ? (u64)bits_of(pack(m << c, top - 1023 - 58 - c)) : 0ull));
}
// 1/x, sqrt(x) and 1/sqrt(x) on the integer pipe (about 36, 45 and 45 instructions) for kernels that FP64 issue
// bounds: 3, 5 and 5 FP64 operations of 64 cycles each.  Rounded from 2^-59; the ranges of recip3 and sqrt3.
__host__ __device__ __forceinline__ u64 significand(u64 b) { return ((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11; }
__host__ __device__ __forceinline__ double recip_fix(double x) {
    const u64 b = (u64)bits_of(x);
    const int ex = (int)(b >> 52) & 0x7FF;
    if ((unsigned)(ex - 2) > 2040u) return 1.0 / x;
    return from_bits((u64)bits_of(pack(recip64(significand(b)), 1023 - ex - 64)) | (b & 0x8000000000000000ull));
}
__host__ __device__ __forceinline__ double sqrt_fix(double x) {
    const u64 b = (u64)bits_of(x);
    const int ex = (int)(b >> 52);  // with the sign: a negative x fails the range test
    if ((unsigned)(ex - 2) > 2040u) return sqrt(x);
    const int X = ex - 1023 - 63, odd = X & 1;
    return pack(sqrt64(significand(b) >> odd) << 1, (X + odd) / 2 - 32);
}
__host__ __device__ __forceinline__ double rsqrt_fix(double x) {
    const u64 b = (u64)bits_of(x);
    const int ex = (int)(b >> 52);
#ifdef __CUDA_ARCH__
    if ((unsigned)(ex - 2) > 2040u) return rsqrt(x);
#endif
    const int X = ex - 1023 - 63, odd = X & 1;
    return pack(rsqrt64(significand(b) >> odd), -95 - (X + odd) / 2);
}


// a / b and sqrt(x) correctly rounded, as the division and the root of IEEE arithmetic are, for code whose
// results must not change: the quotient or root to 2^-58, then its last place decided by the exact remainder
// at the midpoint (of which 64 bits suffice).  About 70 instructions each.
__host__ __device__ __forceinline__ double div_rn(double a, double b) {
    const u64 ba = (u64)bits_of(a), bb = (u64)bits_of(b);
    const int ea = (int)(ba >> 52) & 0x7FF, eb = (int)(bb >> 52) & 0x7FF;
    const u64 sign = (ba ^ bb) & 0x8000000000000000ull;
    const bool zero = (ba << 1) == 0;
    const int e = ea - eb + 1023;
    // normal operands, a quotient safely normal
    if ((unsigned)(eb - 1) > 2045u || (!zero && ((unsigned)(ea - 1) > 2045u || (unsigned)(e - 2) > 2042u))) return a / b;
    const u64 ma = significand(ba) >> 11, mb = significand(bb) >> 11;
    u64 q = umulhi(ma << 11, recip64(mb << 11));  // 2^63 for one
    const int up = (int)((q >> 63) ^ 1);          // below one
    q <<= up;
    u64 n = q >> 11;
    if ((i64)((ma << (53 + up)) - (2 * n + 1) * mb) > 0) ++n;
    return from_bits(sign | (zero ? 0 : ((u64)(e - up - 1) << 52) + n));
}
__host__ __device__ __forceinline__ double sqrt_rn(double x) {
    const u64 b = (u64)bits_of(x);
    const int ex = (int)(b >> 52);  // with the sign
    if ((unsigned)(ex - 2) > 2040u) return sqrt(x);
    const int X = ex - 1023 - 63, odd = X & 1;
    const u64 m = significand(b) >> odd;  // x = m 2^(X + odd), m in [2^62, 2^64)
    u64 n = sqrt64(m) >> 10;              // 2^21 sqrt(m), 53 bits
    // sqrt(m) 2^22 against 2 n + 1: m 2^44 - (2 n + 1)^2
    if ((i64)((m << 44) - (2 * n + 1) * (2 * n + 1)) > 0) ++n;
    return from_bits(((u64)((X + odd) / 2 - 21 + 52 + 1023 - 1) << 52) + n);
}

// the exact conversion float -> double and the rounded one back, which the FP64 pipe would do at its rate; its
// instructions in calls, since predicated they would be issued for nothing
static __device__ __noinline__ double widen_any(float x) { return (double)x; }
static __device__ __noinline__ float narrow_any(double x) { return (float)x; }
__device__ __forceinline__ double widen_fix(float x) {
    const unsigned b = __float_as_uint(x), ex = (b >> 23) & 0xFFu;
    if (ex - 1u > 253u && (b << 1)) return widen_any(x);  // subnormal, infinite or NaN
    return __hiloint2double((int)((b & 0x80000000u) | (ex ? (((b & 0x7FFFFFFFu) >> 3) + (896u << 20)) : 0u)), (int)(b << 29));
}
__device__ __forceinline__ float narrow_fix(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), ex = (hi >> 20) & 0x7FFu;
    if (ex == 0u) return __uint_as_float(hi & 0x80000000u);  // zero, or far below the smallest float
    if (ex - 897u > 253u) return narrow_any(x);  // the result is zero or not a normal float
    const unsigned f = (hi & 0x80000000u) | ((((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29));
    const unsigned r = lo & 0x1FFFFFFFu;
    return __uint_as_float(f + (r > 0x10000000u || (r == 0x10000000u && (f & 1u)) ? 1u : 0u));
}

// in FP64, as a call: inlined it would be predicated, and its operations issued for nothing
static __device__ __noinline__ double sum_differences_fp64(double a1, double a0, double b1, double b0, double c1, double c0) {
    return ((a1 - a0) + (b1 - b0)) + (c1 - c0);
}
// (a1 - a0) + (b1 - b0) + (c1 - c0) from integers in units of 2^-58 of the largest number's power of two, rounded
// once (one FP64 operation, the conversion, for five); not finite or beyond 2^977: in FP64.  Two equal numbers
// cancel exactly and do not count for the units (a uniform pressure would leave a weak shear 2^-58 of itself); their
// shift is then beyond 63 or negative, and both give 0.
__device__ __forceinline__ double sum_differences(double a1, double a0, double b1, double b0, double c1, double c0) {
    int top = 64;
    auto widest = [&](double x, double y) {
        const int e = max((__double2hiint(x) >> 20) & 0x7FF, (__double2hiint(y) >> 20) & 0x7FF);
        top = max(top, bits_of(x) == bits_of(y) && e <= 2000 ? 0 : e);
    };
    widest(a1, a0); widest(b1, b0); widest(c1, c0);
    if (top > 2000) return sum_differences_fp64(a1, a0, b1, b0, c1, c0);
    auto fx = [&](double x) { return to_fixed<6>(bits_of(x), top); };
    return from_fixed(((fx(a1) - fx(a0)) + (fx(b1) - fx(b0))) + (fx(c1) - fx(c0)), top);
}

// (a + b) + (c + d), and 2^-shift of it, in the same way
static __device__ __noinline__ double sum4_fp64(double a, double b, double c, double d, int shift) {
    return ldexp((a + b) + (c + d), -shift);
}
__device__ __forceinline__ double sum4(double a, double b, double c, double d, int shift) {
    int top = 128;
    auto widest = [&](double x) { top = max(top, (__double2hiint(x) >> 20) & 0x7FF); };
    widest(a); widest(b); widest(c); widest(d);
    if (top > 2000) return sum4_fp64(a, b, c, d, shift);
    auto fx = [&](double x) { return to_fixed<6>(bits_of(x), top); };
    return from_fixed((fx(a) + fx(b)) + (fx(c) + fx(d)), top - shift);
}

}  // namespace euler
}  // namespace hype
