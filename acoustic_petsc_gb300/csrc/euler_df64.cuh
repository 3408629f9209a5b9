// euler_df64.cuh -- the CWENO4 reconstruction of euler_kernels.cuh (cweno4) in double-float arithmetic (df64.cuh), for
// the HYPE_PREC_DF64 form of the 3D acoustic solver.
//
// Every coefficient but the constant one is formed from differences of neighbours, on which the 48-bit significand is
// spent.  The coefficients, smoothness indicators and nonlinear weights are the same mathematics as cweno4
// (3d/weno4/Viscous-Multiphase-Fourth-Order/reconstruction.c:38-259); the weights take the ratio form
// w_k = g_k (m / s_k)^4 / sum, m = min_k s_k, s_k = IS_k + 1e-12, because (1e-12)^4 is below the FP32 exponent range.
#pragma once

#include "df64.cuh"
#include "euler_kernels.cuh"

namespace hype {
namespace euler {

__device__ __forceinline__ df64 df_half(df64 x) { return df_scale(x, 0.5f); }
__device__ __forceinline__ df64 df_quarter(df64 x) { return df_scale(x, 0.25f); }

// 20 CWENO4 (or, linear, R4) coefficients of one variable from its 33-point stencil
__device__ __forceinline__ void cweno4_df(const df64* __restrict__ s, bool linear, df64* __restrict__ cf) {
    const df64 u0 = s[0];
    df64 d4[3], dd4[3], ddd4[3], c1[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const df64 m2 = s[S1(d, -2)], m1 = s[S1(d, -1)], p1 = s[S1(d, 1)], p2 = s[S1(d, 2)];
        const df64 a = p1 - m1, b = p2 - m2;
        d4[d] = a * dfc(82. / 120.) - b * dfc(11. / 120.);
        dd4[d] = df_half(m1 + p1) - u0;
        ddd4[d] = (b - df_scale(a, 2.0f)) * dfc(1. / 12.);
        c1[d] = df_half(a);
    }
    df64 cx[3], aab[3], abb[3];
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        const df64 mm = s[SQ(a, 0, b, 0)], mp = s[SQ(a, 0, b, 1)], pm = s[SQ(a, 1, b, 0)], pp = s[SQ(a, 1, b, 1)];
        const df64 Pd = pp - mm, Qd = mp - pm;
        cx[P] = df_quarter((mm + pp) - (mp + pm));
        aab[P] = df_quarter(Pd + Qd) - c1[b];
        abb[P] = df_quarter(Pd - Qd) - c1[a];
    }
    const df64 xyz = df_scale((s[SO(1, 1, 1)] - s[SO(0, 0, 0)]) +
                                  ((s[SO(0, 0, 1)] + s[SO(0, 1, 0)] + s[SO(1, 0, 0)]) -
                                   (s[SO(0, 1, 1)] + s[SO(1, 0, 1)] + s[SO(1, 1, 0)])),
                              0.125f);
    cf[0] = u0;
    if (linear) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            cf[CLIN(d)] = d4[d];
            cf[CSQ(d)] = dd4[d];
            cf[CCUBE(d)] = ddd4[d];
        }
        cf[7] = cx[0]; cf[8] = cx[1]; cf[9] = cx[2];
        cf[13] = aab[0]; cf[14] = abb[0]; cf[15] = aab[1]; cf[16] = abb[1]; cf[17] = aab[2]; cf[18] = abb[2]; cf[19] = xyz;
        return;
    }
    df64 c1sq[3], ddsq[3], cxsq[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        c1sq[d] = df_sqr(c1[d]);
        ddsq[d] = df_sqr(dd4[d]);
        cxsq[d] = df_sqr(cx[d]);
    }
    const df64 r13_3 = dfc(13. / 3.), r7_6 = dfc(7. / 6.);
    const df64 common = (ddsq[0] + ddsq[1] + ddsq[2]) * r13_3 + (cxsq[0] + cxsq[1] + cxsq[2]) * r7_6;
    // sums as balanced trees: a double-float addition is a chain of ~9 dependent FP32
    // operations, so independent partial sums keep more of them in flight
    const df64 lin = (d4[0] * (d4[0] + ddd4[0] * dfc(0.2)) + d4[1] * (d4[1] + ddd4[1] * dfc(0.2))) +
                     (d4[2] * (d4[2] + ddd4[2] * dfc(0.2)) + common);
    const df64 mixed = ((df_sqr(aab[0]) + df_sqr(abb[0])) + (df_sqr(aab[1]) + df_sqr(abb[1]))) +
                       (df_sqr(aab[2]) + df_sqr(abb[2]));
    const df64 cubic = (df_sqr(ddd4[0]) + df_sqr(ddd4[1])) + df_sqr(ddd4[2]);
    const df64 IS4 = (lin + mixed * dfc(4.7)) + (cubic * dfc(39.06) + df_sqr(xyz) * dfc(61. / 48.));
    const df64 IS0 = (c1sq[0] + c1sq[1] + c1sq[2]) + common;
    df64 sd1[6], sd2[6], sx1[6], sx2[6], IS3[6];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int e1 = (d == 0) ? 1 : 0, e2 = (d == 2) ? 1 : 2;
        const int k1 = (d + e1 == 1) ? 0 : (d + e1 == 3) ? 1 : 2;
        const int k2 = (d + e2 == 1) ? 0 : (d + e2 == 3) ? 1 : 2;
        const df64 p1 = s[S1(d, 1)], p2 = s[S1(d, 2)], m1 = s[S1(d, -1)], m2 = s[S1(d, -2)];
        sd2[2 * d] = df_half(u0 + p2) - p1;
        sd1[2 * d] = (p1 - u0) - sd2[2 * d];
        sx1[2 * d] = df_half(s[SQ(d, 1, e1, 1)] - s[SQ(d, 1, e1, 0)]) - c1[e1];
        sx2[2 * d] = df_half(s[SQ(d, 1, e2, 1)] - s[SQ(d, 1, e2, 0)]) - c1[e2];
        sd2[2 * d + 1] = df_half(m2 + u0) - m1;
        sd1[2 * d + 1] = (u0 - m1) + sd2[2 * d + 1];
        sx1[2 * d + 1] = df_half(s[SQ(d, 0, e1, 0)] - s[SQ(d, 0, e1, 1)]) + c1[e1];
        sx2[2 * d + 1] = df_half(s[SQ(d, 0, e2, 0)] - s[SQ(d, 0, e2, 1)]) + c1[e2];
        const int k3 = 3 - k1 - k2;
        const df64 rest1 = c1sq[e1] + c1sq[e2];
        const df64 rest2 = ddsq[e1] + ddsq[e2];
        const df64 restx = cxsq[k3];
#pragma unroll
        for (int sg = 0; sg < 2; ++sg) {
            const int m = 2 * d + sg;
            const df64 a1 = rest1 + df_sqr(sd1[m]);
            const df64 a2 = rest2 + df_sqr(sd2[m]);
            const df64 a3 = restx + df_sqr(sx1[m]) + df_sqr(sx2[m]);
            IS3[m] = a1 + a2 * r13_3 + a3 * r7_6;
        }
    }
    // weights: gammaHi = gammaLo = 0.85, p = 4, eps = 1e-12, in the ratio form
    df64 q[8];
    q[0] = IS4 + dfc(1.0e-12);
    q[1] = IS0 + dfc(1.0e-12);
#pragma unroll
    for (int m = 0; m < 6; ++m) q[2 + m] = IS3[m] + dfc(1.0e-12);
    df64 mn = q[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) mn = df_min(mn, q[k]);
    df64 w[8];
    const df64 gk[3] = {dfc(0.85), dfc((1.0 - 0.85) * 0.85), dfc((1. / 6.) * (1 - 0.85) * (1 - 0.85))};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const df64 r2 = df_sqr(df_div(mn, q[k]));
        w[k] = df_sqr(r2) * gk[k == 0 ? 0 : k == 1 ? 1 : 2];
    }
    const df64 total = ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
    const df64 rt = df_div(dfc(1.0), total);
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = w[k] * rt;
    const df64 wr = w[0] * dfc(1.0 / 0.85);
    const df64 o0 = w[1] - wr * gk[1];
    df64 os[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) os[m] = w[2 + m] - wr * gk[2];
    const df64 ox = os[0] + os[1], oy = os[2] + os[3], oz = os[4] + os[5];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const df64 okeep = o0 + ((d == 0) ? oy + oz : (d == 1) ? ox + oz : ox + oy);
        cf[CLIN(d)] = (wr * d4[d] + okeep * c1[d]) + (os[2 * d] * sd1[2 * d] + os[2 * d + 1] * sd1[2 * d + 1]);
        cf[CSQ(d)] = (wr + okeep) * dd4[d] + (os[2 * d] * sd2[2 * d] + os[2 * d + 1] * sd2[2 * d + 1]);
    }
    cf[7] = (wr + o0 + oz) * cx[0] + ((os[0] * sx1[0] + os[1] * sx1[1]) + (os[2] * sx1[2] + os[3] * sx1[3]));
    cf[8] = (wr + o0 + ox) * cx[1] + ((os[2] * sx2[2] + os[3] * sx2[3]) + (os[4] * sx2[4] + os[5] * sx2[5]));
    cf[9] = (wr + o0 + oy) * cx[2] + ((os[0] * sx2[0] + os[1] * sx2[1]) + (os[4] * sx1[4] + os[5] * sx1[5]));
#pragma unroll
    for (int d = 0; d < 3; ++d) cf[CCUBE(d)] = wr * ddd4[d];
    cf[13] = wr * aab[0]; cf[14] = wr * abb[0]; cf[15] = wr * aab[1]; cf[16] = wr * abb[1];
    cf[17] = wr * aab[2]; cf[18] = wr * abb[2]; cf[19] = wr * xyz;
}

}  // namespace euler
}  // namespace hype
