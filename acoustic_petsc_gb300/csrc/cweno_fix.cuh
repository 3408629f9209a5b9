// cweno_fix.cuh -- the CWENO4 / R4 reconstruction of one FP64 variable and the Rusanov flux's side states on the
// integer pipe.
//
// The mathematics is cweno64.cuh's.  What bounds that form is FP64 issue (fixed.cuh).  A stencil is therefore
// taken to 64-bit fixed point, scaled by the largest magnitude in it (units of 2^-58 of its power of two, 64
// times finer than that number's last FP64 place):
//  * the differences are integer subtractions, exact for values within 2^-6 of the largest;
//  * the smoothness indicators are sums of exact 128-bit products.  With dp, dm the third differences of the
//    one-sided stencils (s2 - D) and c2 = u_ab+ + u_ab-, the indicators of the one-sided stencils differ from
//    the centred one's by dp (8 dp - 3 A + 13 D) and aab (aab +- 2 c2) terms: 37 products for all eight, and
//    the cancellation in them is harmless because it is exact; eps enters through the one they share;
//  * the nonlinear weights are significands with an exponent: one reciprocal and two squarings per indicator;
//  * the weights sum to one, so the combination is R4's centred values plus two corrections per term,
//    o_+ dp, o_- dm and (o_+ - o_-) aab;
//  * the traces are sums of integers with products by fixed-point constants, rounded to FP64 once by the
//    conversion instruction (the FP64 pipe's only work here).
// About 4400 instructions a warp and variable against 361 FP64 ones of 64 cycles.  At 256^3, four stages: all in
// FP64 237.7 ms; integers with the weights in FP64 (67 operations) 80.3; that with products of 32-bit halves
// 76.7; integer weights 73; conversions by instruction 66.4; eps added once 63.0; the FP64 form as a call 61.1; weights
// completed to one 62.4.
// Errors against 128-bit arithmetic, for stencils of a jump with noise beside it: 0.9e-16 of the stencil's largest
// magnitude, where the FP64 form has 2 to 4e-16; and of the traces themselves 5e-16 down to a tenth of it, as the FP64
// form's.  Cells that are quieter than that beside a jump keep the FP64 form, whose errors stay relative to the cell:
// where density, energy or pressure lies four or more binary exponents below its stencil's largest (from a factor 8 to
// 16 on), and where the nonlinear weights leave the polynomial of any variable below 2^-6 of it (faint; up to there
// 3e-15 of the traces; nearer, a few cells of a smooth pulse would take it too, and on a small grid a few decide: 16^3
// 0.78 -> 0.94 ms for eight steps at 2^-4).  With R4 alone a trace holds 1/64 of the largest at least.  Stencils that
// are not finite take the FP64 form too.
#pragma once

#include "cweno64.cuh"

namespace hype {
namespace euler {

// The stencil in fixed point and what the traces need of it (units: 2^(top - 1023 - 58)); doubled differences
// as in Poly64, and cr2 twice its cr
struct PolyFix {
    i64 u0, lin[3], sq[3], cr2[3], ddd[3], aab[3], abb[3], xyz;
    u64 wr;  // w4 / gammaHi, 2^61 for one
    int top;
};

// the largest biased exponent of the stencil, not below 2^-959 (so that every result is a normal number or zero; the
// first cells that a disturbance reaches hold such values, to 2^-1017)
__host__ __device__ __forceinline__ int stencil_top(const double* __restrict__ s) {
    int top = 64;
#pragma unroll
    for (int i = 0; i < 33; ++i) {
        const int e = (int)(bits_of(s[i]) >> 52) & 0x7FF;
        top = e > top ? e : top;
    }
    return top;
}
// whether the fixed-point form applies: finite, results in range, and (strict) the cell's own value at most three
// binary exponents below the largest, a factor of 8 to 16
__host__ __device__ __forceinline__ bool fix_applies(double u0, int top, bool strict) {
    return top <= 2000 && !(strict && (((int)(bits_of(u0) >> 52) & 0x7FF) < top - 3));
}
// whether the polynomial is so much smaller than its stencil (a quiet cell beside a jump: the weights far from linear,
// cell value and limited derivatives below 2^-6 of the largest's power of two) that the stencil's units do not resolve
// it as FP64 does; on the upper words
__host__ __device__ __forceinline__ bool faint(const PolyFix& p) {
    auto mag = [](i64 x) { return (unsigned)((int)(x >> 32) ^ (int)(x >> 63)); };
    const unsigned l = mag(p.lin[0]) | mag(p.lin[1]) | mag(p.lin[2]), q = mag(p.sq[0]) | mag(p.sq[1]) | mag(p.sq[2]),
                   x = mag(p.cr2[0]) | mag(p.cr2[1]) | mag(p.cr2[2]);
    return p.wr < 1ull << 60 && (mag(p.u0) | (l >> 2) | (q >> 3) | (x >> 4)) < 1u << (58 - 6 - 32);
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
    // 24 times cweno64.cuh's indicators, in units of 2^(t - 1023 - 55) squared, t = max(top, 1000): three bits
    // fewer keep every sum below 2^127, and below 2^-23 the differences' 2^-78 is far finer than their
    // comparison with eps = 1e-12 can tell.  eps enters all of them through J1.
    const int t = top > 1000 ? top : 1000;
    const int sh = t - top + 3 < 63 ? t - top + 3 : 63;
    Sum128 J1, m{0, 0}, DD{0, 0}, sA{0, 0}, J[6];
    {
        const int x = -97 - 2 * (t - 1023 - 55);  // 24 * 4e-12 = em 2^x, x <= 59
        constexpr u64 em = 15211807202738752818ull;
        J1 = x > 0 ? Sum128{em >> (64 - x), em << x} : Sum128{0, (x > -64 ? em >> -x : 0) | 1};
    }
    Split x3[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 a_ = A[a] >> sh, d_ = D[a] >> sh, x = p.cr2[a] >> sh, q = p.ddd[a] >> sh;
        const Split as = split(a_), qs = split(q);
        x3[a] = split(x);
        J1 = J1 + times128(split(24 * a_), as) + times128(split(13 * d_), split(8 * d_)) + times128(split(7 * x), x3[a]);
        DD = DD + square128(qs);
        sA = sA + times128(split(8 * q), as);
        const i64 f = dp[a] >> sh, g = dm[a] >> sh, w = 13 * d_, v = 3 * a_;
        const Sum128 P = times128(split(8 * f), split(8 * f + (w - v))), Q = times128(split(8 * g), split(8 * g + (w + v)));
        J[2 * a] = P + P;
        J[2 * a + 1] = Q + Q;
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        const i64 x = 2 * (p.cr2[P] >> sh), f = p.aab[P] >> sh, g = p.abb[P] >> sh;
        const Split f7 = split(7 * f), g7 = split(7 * g);
        m = m + square128(split(f)) + square128(split(g));
        J[2 * a] = J[2 * a] + times128(f7, split(f + x));
        J[2 * a + 1] = J[2 * a + 1] + times128(f7, split(f - x));
        J[2 * b] = J[2 * b] + times128(g7, split(g + x));
        J[2 * b + 1] = J[2 * b + 1] + times128(g7, split(g - x));
    }
    // The nonlinear weights g_k / (IS_k + eps)^4: with IS + eps = m 2^x normalised and y = 2^127 / m, the fourth
    // power y4 = y^4 2^-192 is in [2^60, 2^64) and what the weights share is taken out by the smallest x.
    u64 y4[8];
    int x[8], xm = 1 << 20;
    auto power = [&](int k, Sum128 v) {
        const Norm n = norm128(v);
        u64 y = recip64(n.m);
        y = umulhi(y, y);
        y4[k] = umulhi(y, y);
        x[k] = n.x;
        xm = n.x < xm ? n.x : xm;
    };
    power(1, J1);
#pragma unroll
    for (int k = 0; k < 6; ++k) power(2 + k, J1 + J[k]);
    {
        // + 28.2 m + 26.7 DD - 8 sA + 61/32 xyz^2
        const Sum128 xx = square128(split(p.xyz >> sh)), x3 = scale128(xx, 3);
        const Sum128 x32{x3.hi >> 5, (x3.lo >> 5) | (x3.hi << 59)};
        power(0, (J1 + scale128(m, 28) + part128(m, 3689348814741910323ull)) +
                     (scale128(DD, 27) - part128(DD, 5534023222112865485ull)) + (xx + xx - x32) - sA);
    }
    u64 low = 0;  // an eighth of the one-sided stencils' sum
#pragma unroll
    for (int k = 2; k < 8; ++k) low += shift_by(y4[k] >> 3, 4 * (x[k] - xm));
    // gammaHi = gammaLo = 0.85: g = 0.85, 0.1275, and 0.00375 of each one-sided stencil
    const u64 tot = umulhi(shift_by(y4[0], 4 * (x[0] - xm)), 15679732462653118874ull) + umulhi(shift_by(y4[1], 4 * (x[1] - xm)), 2351959869397967831ull) +
                    umulhi(low, 553402322211286548ull);
    const int z = clz64(tot);
    const u64 rt = recip64(tot << z), rs = umulhi(rt, 17708874310761169551ull);  // 0.00375 2^8 times it
    p.wr = shift_by(umulhi(y4[0], rt), 4 * (x[0] - xm) + 2 - z);
    const u64 sub = umulhi(p.wr, 138350580552821637ull);  // 0.0075
    i64 o[6];  // w_k - wr g_k of the one-sided stencils, 2^62 for one
#pragma unroll
    for (int k = 0; k < 6; ++k) o[k] = (i64)(shift_by(umulhi(y4[2 + k], rs), 4 * (x[2 + k] - xm) + 9 - z) - sub);
    {
        // The weights are off by 2^-57 of each and of their common factor, so their sum by up to 2^-50.  The combination
        // below gives the centred stencil one minus the six; where a jump has suppressed that stencil, the largest of
        // the six takes the difference instead.  o0: the centred stencil's share of w4 / gammaHi and its own weight.
        const i64 o0 = (i64)(2 * umulhi(p.wr, 16094784204311583785ull) +
                             shift_by(umulhi(umulhi(y4[1], rt), 9407839477591871324ull), 4 * (x[1] - xm) + 3 - z));
        i64 rest = (1ll << 62) - o0, most = o0;
        int at = -1;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            rest -= o[k];
            at = o[k] > most ? k : at;
            most = o[k] > most ? o[k] : most;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) o[k] += at == k ? rest : 0;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 f = times62(split(dp[a]), split(o[2 * a])), g = times62(split(dm[a]), split(o[2 * a + 1]));
        p.lin[a] = A[a] - f + g;
        p.sq[a] = D[a] + f + g;
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        p.cr2[P] += times62(split(p.aab[P]), split(o[2 * a] - o[2 * a + 1])) +
                    times62(split(p.abb[P]), split(o[2 * b] - o[2 * b + 1]));
    }
}

// the 24 face traces, numbered as store_traces64 numbers them: put(q, value)
template <class Put>
__host__ __device__ __forceinline__ void traces_fix(const PolyFix& p, Put put) {
    // 2^64 times GPT/2, GPT/8, 1/12, 1/48; and 8 times 1/24, GPT 7/72, GPT/24, 1/192 for wr's 2^61
    constexpr i64 kG2 = 2662558164157085696ll, kG8 = 665639541039271424ll, k12 = 1537228672809129301ll, k48 = 384307168202282325ll;
    const Split wn = split((i64)umulhi(p.wr, 6148914691236517205ull)), wt = split((i64)umulhi(p.wr, 4141757144244355527ull)),
                wm = split((i64)umulhi(p.wr, 1775038776104723797ull)), wo = split((i64)umulhi(p.wr, 768614336404564651ull));
    i64 tan[3], odd[3], even[3], cg[3], cc[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        tan[a] = scaled(p.lin[a], split(kG2)) - scaled(p.ddd[a], wt);
        odd[a] = ((p.lin[a] + 2) >> 2) - scaled(p.ddd[a], wn);
        even[a] = p.u0 + scaled(p.sq[a], split(k12));
        cg[a] = scaled(p.cr2[a], split(kG8));
        cc[a] = scaled(p.cr2[a], split(k48));
    }
    const i64 o12 = scaled(p.xyz, wo);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int t1 = d == 0 ? 1 : 0, t2 = d == 2 ? 1 : 2;
        const i64 m1 = d < t1 ? p.aab[pair_of(d, t1)] : p.abb[pair_of(d, t1)];
        const i64 m2 = d < t2 ? p.aab[pair_of(d, t2)] : p.abb[pair_of(d, t2)];
        const i64 E1 = tan[t1] + scaled(m1, wm), E2 = tan[t2] + scaled(m2, wm);
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
    auto put = [&](int q, i64 v) { C[q * st] = __longlong_as_double(v); };
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        put(a, p.lin[a]);
        put(3 + a, p.sq[a]);
        put(6 + a, p.cr2[a]);
        put(9 + a, p.ddd[a]);
        put(12 + 2 * a, p.aab[a]);
        put(13 + 2 * a, p.abb[a]);
    }
    put(18, p.xyz);
    put(19, p.top);
}

// the 24 traces of one variable's stencil, trace q at T[q * st], and with the fixed-point form not applying
// (fix_applies; faint, where nothing bounds the cell's own value) false and nothing stored
template <bool LINEAR>
__host__ __device__ __forceinline__ bool recon_fix(const double* __restrict__ s, bool strict, double* __restrict__ T, long long st,
                                          PolyFix& p) {
    const int top = stencil_top(s);
    if (!fix_applies(s[0], top, strict)) return false;
    poly_fix<LINEAR>(s, top, p);
    if (!LINEAR && !strict && faint(p)) return false;
    traces_fix(p, [&](int q, double v) { T[q * st] = v; });
    return true;
}

// ---------------------------------------------------------------- Rusanov

// One side of an axis face on the integer pipe: normal velocity, pressure and |u_n| + c from the conserved
// trace (rho, normal, two tangential momenta, E), each to 2^-59 before its rounding to FP64.  Numbers are
// 64-bit significands with an exponent; only sums align.  18 FP64 operations (a reciprocal, a root, 9 products
// and sums) become about 290 integer ones, a third of their issue time.  False (the caller takes the FP64
// form, which also decides on the floors) for a density below 2^-45, a pressure below 2^-38 or not positive,
// and anything not finite or beyond 2^200 (gamma: 2^100).  A normal momentum or velocity that is not a normal number
// (2^-1021 and less, whose exponent has no place in the result) counts as zero.
__host__ __device__ __forceinline__ bool side_fix(double rho, double mn, double m1, double m2, double E, double gamma, double gm1,
                                                  double& un, double& p, double& sp) {
    constexpr u64 FRAC = 0xFFFFFFFFFFFFFull, ONE = 0x10000000000000ull;
    const u64 br = (u64)bits_of(rho), be = (u64)bits_of(E), b0 = (u64)bits_of(mn), b1 = (u64)bits_of(m1), b2 = (u64)bits_of(m2);
    const int xr = (int)(br >> 52), xe = (int)(be >> 52);  // with the sign: a negative one fails the tests
    const int x0 = (int)(b0 >> 52) & 0x7FF, x1 = (int)(b1 >> 52) & 0x7FF, x2 = (int)(b2 >> 52) & 0x7FF;
    const int xm = x0 > x1 ? (x0 > x2 ? x0 : x2) : (x1 > x2 ? x1 : x2);
    if ((unsigned)(xr - (1023 - 45)) > 245u || (unsigned)(xe - (1023 - 100)) > 300u || xm > 1223 ||
        (int)((u64)bits_of(gamma) >> 52) > 1123)
        return false;
    const int er = xr - 1023, ee = xe - 1023, em = xm - 1023;
    const u64 y = recip64(((br & FRAC) | ONE) << 11);  // 1/rho = y 2^(-64 - er)
    // |m|^2 = s 2^(2 em - 58), |m|^2 / (2 rho) = k 2^(2 em - er - 59)
    const u64 q0 = shift_by(((b0 & FRAC) | ONE) << 9, xm - x0), q1 = shift_by(((b1 & FRAC) | ONE) << 9, xm - x1),
              q2 = shift_by(((b2 & FRAC) | ONE) << 9, xm - x2);
    u64 k = umulhi(umulhi(q0, q0) + umulhi(q1, q1) + umulhi(q2, q2), y);
    const int d = 2 * em - er - ee + 2;  // to E's unit 2^(ee - 61)
    if (d > 0 && (d > 30 || (k >> (62 - d)))) return false;
    k = shift_by(k, -d);
    const i64 P0 = (i64)((((be & FRAC) | ONE) << 9) - k);
    if (P0 <= 0) return false;
    const int c0 = clz64((u64)P0);
    const u64 bg = (u64)bits_of(gm1), ba = (u64)bits_of(gamma);
    u64 q = umulhi((u64)P0 << c0, ((bg & FRAC) | ONE) << 11);
    const int u0 = (int)((q >> 63) ^ 1);
    q <<= u0;
    const int xp = ee - 60 - c0 + ((int)(bg >> 52) - 1023) - u0;  // p = q 2^xp
    if (xp < -38 - 63) return false;
    p = pack(q, xp);
    // c^2 = w 2^x
    u64 w = umulhi(umulhi(q, y), ((ba & FRAC) | ONE) << 11);
    int x = xp - er + ((int)(ba >> 52) - 1023) + 1;
    const int c1 = clz64(w);
    w <<= c1;
    x -= c1;
    w >>= x & 1;
    x += x & 1;
    const u64 C = sqrt64(w);  // c = C 2^(x/2 - 31)
    // |u_n| = U 2^(e0 - er - 63)
    const u64 U = x0 ? umulhi(((b0 & FRAC) | ONE) << 11, y) : 0;
    const int u1 = (int)((U >> 63) ^ 1), e0 = x0 - 1023;
    const int least = xr - 1022 > 0 ? xr - 1022 : 0;
    un = from_bits((x0 > least ? (u64)bits_of(pack(U << u1, e0 - er - 63 - u1)) : 0ull) | (b0 & 0x8000000000000000ull));
    const int xu = e0 - er - 62, xc = x / 2 - 31, xs = xu > xc ? xu : xc;
    const u64 S = shift_by(U >> 1, xs - xu) + shift_by(C, xs - xc);
    const int c2 = clz64(S);
    sp = pack(S << c2, xs - c2);
    return true;
}

// rusanov64 with both sides' velocity, pressure and wave speed from the integer pipe: 22 FP64 operations
template <int D>
__device__ __forceinline__ double rusanov_fix(const double* __restrict__ QL, const double* __restrict__ QR, double gamma,
                                              double gm1, double* __restrict__ F, bool& bad) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    double un[2], p[2], sp[2];
    if (!(side_fix(QL[0], QL[1 + D], QL[1 + T1], QL[1 + T2], QL[4], gamma, gm1, un[0], p[0], sp[0]) &&
          side_fix(QR[0], QR[1 + D], QR[1 + T1], QR[1 + T2], QR[4], gamma, gm1, un[1], p[1], sp[1])))
        return rusanov64<D>(QL, QR, gamma, gm1, F, bad);
    const double s = max_pos(sp[0], sp[1]);
    double f[NV];
    f[0] = QL[1 + D] + QR[1 + D];
    const double ps = p[0] + p[1];
#pragma unroll
    for (int i = 1; i < 4; ++i) f[i] = i == 1 + D ? fma(QR[i], un[1], fma(QL[i], un[0], ps)) : fma(QR[i], un[1], QL[i] * un[0]);
    f[4] = fma(QR[4] + p[1], un[1], (QL[4] + p[0]) * un[0]);
#pragma unroll
    for (int c = 0; c < NV; ++c) F[c] = fma(-s, QR[c] - QL[c], f[c]);
    return s;
}

}  // namespace euler
}  // namespace hype
