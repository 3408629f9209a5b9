// cweno_fix.cuh -- the CWENO4 / R4 reconstruction of one FP64 variable on the integer pipe.
//
// The mathematics is cweno64.cuh's.  What bounds that form is FP64 issue: a warp instruction holds the
// FP64 pipe for 64 cycles of its scheduler, a 64-bit integer addition for 2 and a 64 x 64 bit product's
// upper half for 17 (measured).  A stencil is therefore taken to 64-bit fixed point, scaled by the largest
// magnitude in it (units of 2^-58 of its power of two, 64 times finer than that number's last FP64 place):
//  * the differences are integer subtractions, exact for values within 2^-6 of the largest;
//  * the smoothness indicators are sums of exact 128-bit products, rounded once.  With dp, dm the
//    third differences of the one-sided stencils (s2 - D) and c2 = u_ab+ + u_ab-, the indicators of the
//    one-sided stencils differ from the centred one's by dp (8 dp - 3 A + 13 D) and aab (aab +- 2 c2)
//    terms: 34 products for all eight, and the cancellation in them is harmless because it is exact;
//  * the nonlinear weights (two powers, nine reciprocals) stay in FP64: 67 operations;
//  * the weights sum to one, so the combination is R4's centred values plus two corrections per term,
//    o_+ dp, o_- dm and (o_+ - o_-) aab;
//  * the traces are sums of integers with products by fixed-point constants, rounded to FP64 once.
// Errors: 2^-57 of the stencil's largest magnitude, where the FP64 form has a few 2^-53.  A cell whose own
// value is more than 8 times below the largest of its stencil (a strong shock in density, energy or
// pressure) or whose stencil is not finite keeps the FP64 form, whose error there is relative to the cell.
#pragma once

#include <string.h>

#include "cweno64.cuh"

namespace hype {
namespace euler {

typedef unsigned long long u64;
typedef long long i64;
typedef unsigned __int128 u128;
typedef __int128 i128;

__host__ __device__ __forceinline__ u64 umulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((u128)a * b) >> 64);
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
__host__ __device__ __forceinline__ u128 sqr(i64 a) { return (u128)((i128)a * a); }
__host__ __device__ __forceinline__ i128 prod(i64 a, i64 b) { return (i128)a * b; }

// x * c / 2^64 for an unsigned multiplier, rounded to the nearest
__host__ __device__ __forceinline__ i64 scale_u(i64 x, u64 c) {
    return (i64)(umulhi((u64)x, c) - (x < 0 ? c : 0ull));
}

// a finite double with biased exponent e <= top as an integer: 2^(52 + SHIFT) stands for 2^(top - 1023)
template <int SHIFT>
__host__ __device__ __forceinline__ i64 to_fixed(i64 b, int top) {
    const int e = (int)(b >> 52) & 0x7FF;
    const u64 m = ((b & 0xFFFFFFFFFFFFFll) | 0x10000000000000ll) << SHIFT;
    const int sh = top - e;
    const i64 v = (i64)(m >> (sh < 63 ? sh : 63));
    const i64 s = b >> 63;
    return (v ^ s) - s;
}
// v * 2^(top - 1023 - 58) rounded to the nearest double; the result's exponent is in range by the clamp of top
__host__ __device__ __forceinline__ double from_fixed(i64 v, int top) {
    const i64 s = v >> 63;
    const u64 m = (u64)((v ^ s) - s);
    if (m == 0) return 0.0;
    const int c = clz64(m);
    const u64 t = m << c;
    const u64 r = (t >> 11) + ((t >> 10) & 1);
    return from_bits(((u64)(s & 1) << 63) | (((u64)(top + 5 - c - 1) << 52) + r));
}
// J * 2^e2 rounded to a double (0 for 0)
__host__ __device__ __forceinline__ double from_u128(u128 J, int e2) {
    u64 hi = (u64)(J >> 64), lo = (u64)J;
    int n = 0;
    if (hi == 0) {
        hi = lo;
        lo = 0;
        n = 64;
    }
    if (hi == 0) return 0.0;
    const int c = clz64(hi);
    const u64 t = (hi << c) | ((lo >> 1) >> (63 - c));
    const u64 r = (t >> 11) + ((t >> 10) & 1);
    return from_bits(((u64)(1023 + 127 - n - c + e2 - 1) << 52) + r);
}

// The stencil in fixed point and what the traces need of it (units: 2^(top - 1023 - 58)); doubled differences
// as in Poly64, and cr2 twice its cr
struct PolyFix {
    i64 u0, lin[3], sq[3], cr2[3], ddd[3], aab[3], abb[3], xyz;
    u64 wr;  // w4 / gammaHi, 2^61 for one
    int top;
};

// the largest biased exponent of the stencil, not below 2^-400 (smaller numbers become zero)
__host__ __device__ __forceinline__ int stencil_top(const double* __restrict__ s) {
    int top = 623;
#pragma unroll
    for (int i = 0; i < 33; ++i) {
        const int e = (int)(bits_of(s[i]) >> 52) & 0x7FF;
        top = e > top ? e : top;
    }
    return top;
}
// whether the fixed-point form applies: finite, no overflow of the indicators, and (strict) the cell's own
// value within a factor 8 of the largest
__host__ __device__ __forceinline__ bool fix_applies(double u0, int top, bool strict) {
    return top <= 1423 && !(strict && (((int)(bits_of(u0) >> 52) & 0x7FF) < top - 3));
}

template <bool LINEAR>
__host__ __device__ __forceinline__ void poly_fix(const double* __restrict__ s, int top, PolyFix& p) {
    i64 A[3], D[3], dp[3], dm[3];
    auto v = [&](int i) { return to_fixed<6>(bits_of(s[i]), top); };
    p.top = top;
    const i64 u0 = v(0);
    p.u0 = u0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 p1 = v(S1(a, 1)), m1 = v(S1(a, -1)), p2 = v(S1(a, 2)), m2 = v(S1(a, -2));
        const i64 ep = p1 - u0, em = u0 - m1;
        A[a] = p1 - m1;
        D[a] = ep - em;
        dp[a] = (p2 - p1) - ep - D[a];
        dm[a] = em - (m1 - m2) - D[a];
        p.ddd[a] = dp[a] - dm[a];
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        const i64 mm = v(SQ(a, 0, b, 0)), mp = v(SQ(a, 0, b, 1)), pm = v(SQ(a, 1, b, 0)), pp = v(SQ(a, 1, b, 1));
        const i64 d = pp - mm, x = mp - pm;
        p.cr2[P] = (pp + mm) - (mp + pm);
        p.aab[P] = d + x - 2 * A[b];
        p.abb[P] = d - x - 2 * A[a];
    }
    p.xyz = ((v(SO(1, 1, 1)) - v(SO(0, 0, 0))) + (v(SO(0, 0, 1)) - v(SO(1, 1, 0)))) +
            ((v(SO(0, 1, 0)) - v(SO(1, 0, 1))) + (v(SO(1, 0, 0)) - v(SO(0, 1, 1))));
    if (LINEAR) {
        p.wr = 1ull << 61;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            p.lin[a] = A[a];
            p.sq[a] = D[a];
        }
        return;
    }
    // 24 times cweno64.cuh's indicators, in units of 2^(top - 1023 - 55) squared: three bits fewer keep every
    // sum below 2^127
    u128 J1 = 0, m = 0, DD = 0, J[6];
    i128 sA = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 a_ = A[a] >> 3, d_ = D[a] >> 3, x = p.cr2[a] >> 3, q = p.ddd[a] >> 3;
        J1 += 24 * sqr(a_) + 104 * sqr(d_) + 7 * sqr(x);
        DD += sqr(q);
        sA += prod(q, a_);
        const i64 f = dp[a] >> 3, g = dm[a] >> 3;
        J[2 * a] = (u128)(16 * prod(f, 8 * f - 3 * a_ + 13 * d_));
        J[2 * a + 1] = (u128)(16 * prod(g, 8 * g + 3 * a_ + 13 * d_));
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        const i64 x = p.cr2[P] >> 3, f = p.aab[P] >> 3, g = p.abb[P] >> 3;
        const u128 ff = sqr(f), gg = sqr(g);
        const i128 fx = 2 * prod(f, x), gx = 2 * prod(g, x);
        m += ff + gg;
        J[2 * a] += 7 * (ff + (u128)fx);
        J[2 * a + 1] += 7 * (ff - (u128)fx);
        J[2 * b] += 7 * (gg + (u128)gx);
        J[2 * b + 1] += 7 * (gg - (u128)gx);
    }
    const int e2 = 2 * (top - 1023 - 55);
    constexpr double eps = 24 * 4.0e-12;
    double is[8];
    is[1] = from_u128(J1, e2) + eps;
#pragma unroll
    for (int k = 0; k < 6; ++k) is[2 + k] = from_u128(J1 + J[k], e2) + eps;
    {
        // + 28.2 m + 26.7 DD - 8 sA + 61/32 xyz^2
        const u128 xx = sqr(p.xyz >> 3);
        auto part = [](u128 x, u64 c) { return (u128)(u64)(x >> 64) * c + umulhi((u64)x, c); };  // x c / 2^64
        u128 v4 = J1 + 28 * m + part(m, 3689348814741910323ull) + 27 * DD - part(DD, 5534023222112865485ull) -
                  (u128)(8 * sA) + 2 * xx - ((3 * xx) >> 5);
        is[0] = from_u128(v4, e2) + eps;
    }
    // weights, as cweno64.cuh forms them
    constexpr double g0 = (1.0 - 0.85) * 0.85, gs = (1. / 6.) * (1 - 0.85) * (1 - 0.85);
    double r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#ifdef __CUDA_ARCH__
        r[k] = recip3(is[k]);
#else
        r[k] = 1.0 / is[k];
#endif
        r[k] *= r[k];
        r[k] *= r[k];
    }
    const double low = ((r[2] + r[3]) + (r[4] + r[5])) + (r[6] + r[7]);
    const double tot = fma(gs, low, fma(g0, r[1], 0.85 * r[0]));
#ifdef __CUDA_ARCH__
    const double rt = recip3(tot);
#else
    const double rt = 1.0 / tot;
#endif
    const double wr = r[0] * rt, sc = gs * rt, sub = gs * wr;
    p.wr = (u64)to_fixed<10>(bits_of(wr), 1024);
    i64 o[6];  // w_k - wr g_k of the one-sided stencils, 2^61 for one
#pragma unroll
    for (int k = 0; k < 6; ++k) o[k] = to_fixed<10>(bits_of(fma(sc, r[2 + k], -sub)), 1024);
    // x o, o in units of 2^-61
    auto times = [](i64 x, i64 w) { return (i64)((prod(x, w) + ((i128)1 << 60)) >> 61); };
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 f = times(dp[a], o[2 * a]), g = times(dm[a], o[2 * a + 1]);
        p.lin[a] = A[a] - f + g;
        p.sq[a] = D[a] + f + g;
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        p.cr2[P] += times(p.aab[P], o[2 * a] - o[2 * a + 1]) + times(p.abb[P], o[2 * b] - o[2 * b + 1]);
    }
}

// x c, c in units of 2^-(64 + SH), rounded
template <int SH>
__host__ __device__ __forceinline__ i64 scaled(i64 x, u64 c) {
    return (scale_u(x, c) + (1ll << (SH - 1))) >> SH;
}

// the 24 face traces, numbered as store_traces64 numbers them: put(q, value)
template <class Put>
__host__ __device__ __forceinline__ void traces_fix(const PolyFix& p, Put put) {
    constexpr u64 kG2 = 5325116328314171392ull, kG8 = 5325116328314171392ull;  // GPT/2 2^65, GPT/8 2^67
    constexpr u64 k12 = 6148914691236517205ull, k48 = 6148914691236517205ull;  // 2^66/12, 2^68/48
    constexpr u64 k23 = 12297829382473034411ull;                          // 2^64 2/3
    constexpr u64 kwt = 16567028576977422108ull, kwm = 14200310208837790379ull;  // 2^64 times 2^5 GPT 7/72 and 2^6 GPT/24
    // w4/gammaHi times 1/24 (2^67 for one), GPT 7/72 (2^67), GPT/24 (2^68) and 1/192 (2^70)
    const u64 w23 = umulhi(p.wr, k23) << 2;
    const u64 wn = w23, wo = w23, wt = umulhi(p.wr, kwt) << 1, wm = umulhi(p.wr, kwm) << 1;
    i64 tan[3], odd[3], even[3], cg[3], cc[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        tan[a] = scaled<1>(p.lin[a], kG2) - scaled<3>(p.ddd[a], wt);
        odd[a] = ((p.lin[a] + 2) >> 2) - scaled<3>(p.ddd[a], wn);
        even[a] = p.u0 + scaled<2>(p.sq[a], k12);
        cg[a] = scaled<3>(p.cr2[a], kG8);
        cc[a] = scaled<4>(p.cr2[a], k48);
    }
    const i64 o12 = scaled<6>(p.xyz, wo);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int t1 = d == 0 ? 1 : 0, t2 = d == 2 ? 1 : 2;
        const i64 m1 = d < t1 ? p.aab[pair_of(d, t1)] : p.abb[pair_of(d, t1)];
        const i64 m2 = d < t2 ? p.aab[pair_of(d, t2)] : p.abb[pair_of(d, t2)];
        const i64 E1 = tan[t1] + scaled<4>(m1, wm), E2 = tan[t2] + scaled<4>(m2, wm);
        const i64 c1 = cg[pair_of(d, t1)], c2 = cg[pair_of(d, t2)], c12 = cc[pair_of(t1, t2)];
#pragma unroll
        for (int sn = 0; sn < 2; ++sn) {
            const i64 A = sn ? even[d] + odd[d] : even[d] - odd[d];
            const i64 B1 = sn ? E1 + c1 : E1 - c1, B2 = sn ? E2 + c2 : E2 - c2, B12 = sn ? c12 + o12 : c12 - o12;
            const i64 am = A - B1, ap = A + B1, bm = B2 - B12, bp = B2 + B12;
            put(8 * d + 4 * sn + 0, from_fixed(am - bm, p.top));
            put(8 * d + 4 * sn + 1, from_fixed(am + bm, p.top));
            put(8 * d + 4 * sn + 2, from_fixed(ap - bp, p.top));
            put(8 * d + 4 * sn + 3, from_fixed(ap + bp, p.top));
        }
    }
}

// How far the polynomial can be from its cell value at points with |x| <= 1/2 (basis functions at most 1/2,
// 1/6, 1/4, 1/20, 1/12 and 1/8): an upper bound in the polynomial's units
__device__ __forceinline__ u64 spread_fix(const PolyFix& p) {
    auto mag = [](i64 x) { return (u64)(x < 0 ? -x : x); };
    const u64 l = (mag(p.lin[0]) >> 2) + (mag(p.lin[1]) >> 2) + (mag(p.lin[2]) >> 2);
    const u64 q = (mag(p.sq[0]) >> 3) + (mag(p.sq[1]) >> 3) + (mag(p.sq[2]) >> 3);
    const u64 x = (mag(p.cr2[0]) >> 4) + (mag(p.cr2[1]) >> 4) + (mag(p.cr2[2]) >> 4);
    const u64 c = (mag(p.ddd[0]) >> 4) + (mag(p.ddd[1]) >> 4) + (mag(p.ddd[2]) >> 4) + (mag(p.xyz) >> 6);
    const u64 m = (mag(p.aab[0]) >> 5) + (mag(p.abb[0]) >> 5) + (mag(p.aab[1]) >> 5) + (mag(p.abb[1]) >> 5) +
                  (mag(p.aab[2]) >> 5) + (mag(p.abb[2]) >> 5);
    return l + q + x + (umulhi(c + m, p.wr) << 3) + 64;
}
// the polynomial exceeds lo > 0 at all those points (decided with a margin of 2^-29 of the cell value)
__device__ __forceinline__ bool surely_above(const PolyFix& p, double lo) {
    const i64 low = p.u0 - (p.u0 >> 29) - (i64)spread_fix(p);
    return low > 0 && from_fixed(low, p.top) > lo;
}

// the R4 differences that the viscous fluxes take, as the Poly64 form of store_grad_coeffs stores them
__device__ __forceinline__ void store_grad_coeffs(const PolyFix& p, double* __restrict__ C, long long st) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        C[a * st] = from_fixed(p.lin[a], p.top);
        C[(3 + a) * st] = from_fixed(p.sq[a], p.top);
        C[(6 + a) * st] = from_fixed(p.cr2[a], p.top - 1);
        C[(9 + a) * st] = from_fixed(p.ddd[a], p.top);
        C[(12 + 2 * a) * st] = from_fixed(p.aab[a], p.top);
        C[(13 + 2 * a) * st] = from_fixed(p.abb[a], p.top);
    }
    C[18 * st] = from_fixed(p.xyz, p.top);
}

// the 24 traces of one variable's stencil, trace q at T[q * st], and with the fixed-point form not applying
// (fix_applies) false and nothing stored
template <bool LINEAR>
__device__ __forceinline__ bool recon_fix(const double* __restrict__ s, bool strict, double* __restrict__ T, long long st,
                                          PolyFix& p) {
    const int top = stencil_top(s);
    if (!fix_applies(s[0], top, strict)) return false;
    poly_fix<LINEAR>(s, top, p);
    traces_fix(p, [&](int q, double v) { T[q * st] = v; });
    return true;
}

}  // namespace euler
}  // namespace hype
