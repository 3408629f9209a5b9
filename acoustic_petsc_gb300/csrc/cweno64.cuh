// cweno64.cuh -- the FP64 CWENO4 / R4 reconstruction of one variable and its face traces, the FP64
// Rusanov flux and the viscous fluxes of the 3D solvers.
//
// The mathematics is the reference's (weno(), 3d/weno4/Viscous-Multiphase-Fourth-Order/
// reconstruction.c:38-259; evaluate_polynomial :12-21; PDEConsFlux and LLF,
// 3d/weno4/Navier-Stokes-3D/pde.c:40-88, 164-187).  FP64 issue bounds every kernel that uses it (one
// warp instruction takes 64 issue slots of its scheduler), so the form is chosen by its count of FP64
// operations, with comparisons, maxima and exponent handling on the integer pipe:
//  * everything is built from neighbour differences, doubled where that saves a halving: per axis the
//    inner and outer one-sided differences give the first and second derivatives of R4, of the centred
//    and of the two one-sided quadratics (12 operations); per pair of axes the four edge differences
//    give all four one-sided cross terms, and their sums and differences the centred cross term and the
//    two mixed cubic ones (12);
//  * IS of R4 is IS of the centred quadratic plus a quadratic form in the cubic terms;
//  * 1e-12 enters the indicators through a square sum that each of them contains;
//  * the weights take one 3-operation reciprocal each and only their ratios to the R4 weight;
//  * the R4 cubic terms are scaled by w4/gammaHi inside the trace constants, the basis functions that
//    vanish at the 2x2 Gauss points (GPT^2 = 1/12) are left out, and the products shared by the two
//    directions an axis is tangential to are formed once.
// 361 FP64 operations for a variable's 24 traces (137 for R4 alone) against 470 (194) for the
// coefficient-by-coefficient form, whose rounding it does not exceed: differences of neighbours are
// exact where they lie within a factor 2.
#pragma once

#include "euler_kernels.cuh"
#include "fixed.cuh"

namespace hype {
namespace euler {

// One variable's polynomial.  With c the coefficients of evaluate_polynomial's basis:
//   c_a = lin/2 - wr (11/120) ddd, c_aa = sq/2, c_ab = cr/2, c_aaa = wr ddd/12, c_aab = wr aab/4,
//   c_abb = wr abb/4, c_xyz = wr xyz/8
struct Poly64 {
    double u0, wr;            // cell value; w4 / gammaHi (1 for R4)
    double lin[3], sq[3], cr[3];  // cr: pairs xy, yz, xz
    double ddd[3], aab[3], abb[3], xyz;
};

// the doubled differences R4's terms are made of, and (one-sided ones) those of the R3 stencils
struct Diff64 {
    double A[3], D[3], cx[3];                  // 2 u_a, 2 u_aa, 2 u_ab (centred)
    double t[6], s2[6], x1[6], x2[6];          // one-sided: 2 u_a, 2 u_aa, 2 u_ab with the lower and higher other axis
};

template <bool ONE_SIDED>
__device__ __forceinline__ void diffs64(const double* __restrict__ s, Diff64& d, Poly64& p) {
    const double u0 = s[0];
    p.u0 = u0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double ep = s[S1(a, 1)] - u0, em = u0 - s[S1(a, -1)];
        const double fp = s[S1(a, 2)] - s[S1(a, 1)], fm = s[S1(a, -1)] - s[S1(a, -2)];
        d.A[a] = ep + em;
        d.D[a] = ep - em;
        p.ddd[a] = (fp + fm) - d.A[a];
        if (ONE_SIDED) {
            d.s2[2 * a] = fp - ep;
            d.s2[2 * a + 1] = em - fm;
            d.t[2 * a] = fma(2.0, ep, -d.s2[2 * a]);
            d.t[2 * a + 1] = fma(2.0, em, d.s2[2 * a + 1]);
        }
    }
#pragma unroll
    for (int P = 0; P < 3; ++P) {
        const int a = P == 1 ? 1 : 0, b = P == 0 ? 1 : 2;
        const double mm = s[SQ(a, 0, b, 0)], mp = s[SQ(a, 0, b, 1)], pm = s[SQ(a, 1, b, 0)], pp = s[SQ(a, 1, b, 1)];
        if (!ONE_SIDED) {
            const double dp = pp - pm, dm = mp - mm;
            d.cx[P] = 0.5 * (dp - dm);
            p.aab[P] = fma(-2.0, d.A[b], dp + dm);
            p.abb[P] = fma(-2.0, d.A[a], (pp - mp) + (pm - mm));
            continue;
        }
        // towards +a, -a, +b, -b
        const double ap = (pp - pm) - d.A[b], am = d.A[b] - (mp - mm);
        const double bp = (pp - mp) - d.A[a], bm = d.A[a] - (pm - mm);
        d.cx[P] = 0.5 * (ap + am);
        p.aab[P] = ap - am;
        p.abb[P] = bp - bm;
        // slots of the pair: the other axes of a in increasing order, likewise of b
        if (P == 0) {
            d.x1[0] = ap; d.x1[1] = am; d.x1[2] = bp; d.x1[3] = bm;
        } else if (P == 1) {
            d.x2[2] = ap; d.x2[3] = am; d.x2[4] = bp; d.x2[5] = bm;
        } else {
            d.x2[0] = ap; d.x2[1] = am; d.x1[4] = bp; d.x1[5] = bm;
        }
    }
    p.xyz = ((s[SO(1, 1, 1)] - s[SO(0, 0, 0)]) + ((s[SO(0, 0, 1)] - s[SO(0, 1, 1)]) + (s[SO(0, 1, 0)] - s[SO(1, 0, 1)]))) +
            (s[SO(1, 0, 0)] - s[SO(1, 1, 0)]);
}

__device__ __forceinline__ void r4_64(const double* __restrict__ s, Poly64& p) {
    Diff64 d;
    diffs64<false>(s, d, p);
    p.wr = 1.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p.lin[a] = d.A[a];
        p.sq[a] = d.D[a];
        p.cr[a] = d.cx[a];
    }
}

__device__ __forceinline__ void cweno4_64(const double* __restrict__ s, Poly64& p) {
    Diff64 d;
    diffs64<true>(s, d, p);
    constexpr double r13_3 = 13. / 3., r7_6 = 7. / 6.;
    // four times the indicators, with 4 eps = 4e-12 (half of it in each A^2, of which a one-sided
    // stencil keeps two and the centred one three)
    double Aq[3], Dq[3], Xq[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        Aq[a] = fma(d.A[a], d.A[a], 2.0e-12);
        Dq[a] = d.D[a] * d.D[a];
        Xq[a] = d.cx[a] * d.cx[a];
    }
    const double A2[3] = {Aq[1] + Aq[2], Aq[0] + Aq[2], Aq[0] + Aq[1]};
    const double D2[3] = {Dq[1] + Dq[2], Dq[0] + Dq[2], Dq[0] + Dq[1]};
    double is[8];
    is[1] = (A2[2] + Aq[2]) + fma(r13_3, D2[2] + Dq[2], fma(r7_6, (Xq[0] + Xq[1]) + Xq[2], -2.0e-12));
    {
        double m = p.aab[0] * p.aab[0];
        m = fma(p.abb[0], p.abb[0], m);
        m = fma(p.aab[1], p.aab[1], m);
        m = fma(p.abb[1], p.abb[1], m);
        m = fma(p.aab[2], p.aab[2], m);
        m = fma(p.abb[2], p.abb[2], m);
        double v = fma(1.175, m, is[1]);
        v = fma((61. / 768.) * p.xyz, p.xyz, v);
#pragma unroll
        for (int a = 0; a < 3; ++a) v = fma(p.ddd[a], fma(1.1125, p.ddd[a], (-1. / 3.) * d.A[a]), v);
        is[0] = v;
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const int a = m >> 1, k3 = a == 0 ? 1 : a == 1 ? 2 : 0;  // the pair without axis a
        const double v1 = fma(d.t[m], d.t[m], A2[a]);
        const double v2 = fma(d.s2[m], d.s2[m], D2[a]);
        const double v3 = fma(d.x2[m], d.x2[m], fma(d.x1[m], d.x1[m], Xq[k3]));
        is[2 + m] = fma(r7_6, v3, fma(r13_3, v2, v1));
    }
    // weights g / (IS + eps)^4 (gammaHi = gammaLo = 0.85), as ratios: the common factor cancels
    constexpr double g0 = (1.0 - 0.85) * 0.85, gs = (1. / 6.) * (1 - 0.85) * (1 - 0.85);
    double r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        r[k] = recip3(is[k]);
        r[k] *= r[k];
        r[k] *= r[k];
    }
    const double low = ((r[2] + r[3]) + (r[4] + r[5])) + (r[6] + r[7]);
    const double rt = recip3(fma(gs, low, fma(g0, r[1], 0.85 * r[0])));
    const double wr = r[0] * rt;  // w4 / gammaHi
    const double sc = gs * rt, sub = gs * wr;
    double o[6];  // w_k - wr g_k of the one-sided stencils
#pragma unroll
    for (int m = 0; m < 6; ++m) o[m] = fma(sc, r[2 + m], -sub);
    const double o0 = fma(g0, fma(r[1], rt, -wr), wr);  // wr + (w_0 - wr g_0)
    const double ox = o[0] + o[1], oy = o[2] + o[3], oz = o[4] + o[5];
    const double keep[3] = {o0 + (oy + oz), o0 + (ox + oz), o0 + (ox + oy)};
    p.wr = wr;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p.lin[a] = fma(o[2 * a + 1], d.t[2 * a + 1], fma(o[2 * a], d.t[2 * a], keep[a] * d.A[a]));
        p.sq[a] = fma(o[2 * a + 1], d.s2[2 * a + 1], fma(o[2 * a], d.s2[2 * a], keep[a] * d.D[a]));
    }
    p.cr[0] = fma(o[3], d.x1[3], fma(o[2], d.x1[2], fma(o[1], d.x1[1], fma(o[0], d.x1[0], (o0 + oz) * d.cx[0]))));
    p.cr[1] = fma(o[5], d.x2[5], fma(o[4], d.x2[4], fma(o[3], d.x2[3], fma(o[2], d.x2[2], (o0 + ox) * d.cx[1]))));
    p.cr[2] = fma(o[5], d.x1[5], fma(o[4], d.x1[4], fma(o[1], d.x2[1], fma(o[0], d.x2[0], (o0 + oy) * d.cx[2]))));
}

// the products of a Poly64 that its three directions' traces share
struct Shared64 {
    double tan[3];    // value of t's odd terms at t = GPT without those in x_D^2 t
    double wm, wn;    // wr GPT/24 (of aab), -wr/24 (of ddd)
    double o12;       // c_xyz GPT^2 / 2
};

__device__ __forceinline__ void shared64(const Poly64& p, Shared64& h) {
    const double wt = p.wr * (-GPT * (7. / 72.));
    h.wm = p.wr * (GPT / 24.);
    h.wn = p.wr * (-1. / 24.);
    h.o12 = (p.wr * (1. / 192.)) * p.xyz;
#pragma unroll
    for (int a = 0; a < 3; ++a) h.tan[a] = fma(wt, p.ddd[a], (0.5 * GPT) * p.lin[a]);
}

// the 8 traces of the two faces normal to D, as face_traces: out[4 sn + 2 (t1 > 0) + (t2 > 0)]
template <int D>
__device__ __forceinline__ void traces64(const Poly64& p, const Shared64& h, double* __restrict__ out) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    // x_D^2 t of the pair (D, t): aab where D is the pair's first axis
    const double m1 = D < T1 ? p.aab[pair_of(D, T1)] : p.abb[pair_of(D, T1)];
    const double m2 = D < T2 ? p.aab[pair_of(D, T2)] : p.abb[pair_of(D, T2)];
    const double E0 = fma(1. / 12., p.sq[D], p.u0);
    const double O0 = fma(h.wn, p.ddd[D], 0.25 * p.lin[D]);
    const double E1 = fma(h.wm, m1, h.tan[T1]), E2 = fma(h.wm, m2, h.tan[T2]);
    const double c1 = p.cr[pair_of(D, T1)], c2 = p.cr[pair_of(D, T2)], c12 = p.cr[pair_of(T1, T2)];
#pragma unroll
    for (int sn = 0; sn < 2; ++sn) {
        const double sg = sn ? 1.0 : -1.0;
        const double A = sn ? E0 + O0 : E0 - O0;
        const double B1 = fma(sg * (GPT / 4.), c1, E1);
        const double B2 = fma(sg * (GPT / 4.), c2, E2);
        const double B12 = fma(1. / 24., c12, sn ? h.o12 : -h.o12);
        const double am = A - B1, ap = A + B1;
        const double bm = B2 - B12, bp = B2 + B12;
        out[4 * sn + 0] = am - bm;
        out[4 * sn + 1] = am + bm;
        out[4 * sn + 2] = ap - bp;
        out[4 * sn + 3] = ap + bp;
    }
}

// the 24 face traces of one variable, trace q (8 D + 4 (high side) + 2 (t1 > 0) + (t2 > 0)) at T[q * st]
__device__ __forceinline__ void store_traces64(const Poly64& p, double* __restrict__ T, long long st) {
    Shared64 h;
    shared64(p, h);
    double tr[8];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d == 0) traces64<0>(p, h, tr);
        else if (d == 1) traces64<1>(p, h, tr);
        else traces64<2>(p, h, tr);
#pragma unroll
        for (int q = 0; q < 8; ++q) T[(8 * d + q) * st] = tr[q];
    }
}

// the 20 coefficients in evaluate_polynomial's order, for callers that evaluate it elsewhere
__device__ __forceinline__ void coeffs64(const Poly64& p, double* __restrict__ cf) {
    cf[0] = p.u0;
    const double w3 = p.wr * (1. / 12.), w2 = p.wr * 0.25;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        cf[CCUBE(a)] = w3 * p.ddd[a];
        cf[CLIN(a)] = fma(-1.1, cf[CCUBE(a)], 0.5 * p.lin[a]);
        cf[CSQ(a)] = 0.5 * p.sq[a];
        cf[7 + a] = 0.5 * p.cr[a];
    }
    cf[13] = w2 * p.aab[0]; cf[14] = w2 * p.abb[0]; cf[15] = w2 * p.aab[1]; cf[16] = w2 * p.abb[1];
    cf[17] = w2 * p.aab[2]; cf[18] = w2 * p.abb[2]; cf[19] = (p.wr * 0.125) * p.xyz;
}

// Rusanov across an axis face of normal D without the factor 1/2 (the caller folds it into its
// quadrature weight): F(L) + F(R) - s (Q_R - Q_L); returns s, flags a state below the floors of
// pde.c:56-66.  63 FP64 operations: the floors and the larger speed are decided on bit patterns.
template <int D>
__device__ __forceinline__ double rusanov64(const double* __restrict__ QL, const double* __restrict__ QR, double gamma,
                                            double gm1, double* __restrict__ F, bool& bad) {
    double un[2], p[2], sp[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double* Q = k ? QR : QL;
        const double ir = recip3(Q[0]);
        un[k] = Q[1 + D] * ir;
        const double m2 = fma(Q[3], Q[3], fma(Q[2], Q[2], Q[1] * Q[1]));
        p[k] = gm1 * fma(-0.5, m2 * ir, Q[4]);
        bad |= !(at_least(Q[0], 1.0e-14) && at_least(p[k], 1.0e-12));
        sp[k] = fabs(un[k]) + sqrt3(gamma * p[k] * ir);
    }
    const double s = max_pos(sp[0], sp[1]);
    const double ps = p[0] + p[1];
    double f[NV];
    f[0] = QL[1 + D] + QR[1 + D];
#pragma unroll
    for (int i = 1; i < 4; ++i) f[i] = i == 1 + D ? fma(QR[i], un[1], fma(QL[i], un[0], ps)) : fma(QR[i], un[1], QL[i] * un[0]);
    f[4] = fma(QR[4] + p[1], un[1], (QL[4] + p[0]) * un[0]);
#pragma unroll
    for (int c = 0; c < NV; ++c) F[c] = fma(-s, QR[c] - QL[c], f[c]);
    return s;
}

// ---------------------------------------------------------------- viscous fluxes
// The R4 differences that a cell's gradients need, kept for the face kernel in fixed point (units of
// 2^(top - 1023 - 58)): A, D, 4 u_ab (xy, yz, xz), ddd, then aab and abb by pair, xyz, and top (r4_64's lin, sq,
// twice its cr, ddd, aab/abb, xyz)
__device__ __forceinline__ void store_grad_coeffs(const Poly64& p, double* __restrict__ C, long long st) {
    const double v[19] = {p.lin[0], p.lin[1], p.lin[2], p.sq[0], p.sq[1], p.sq[2], 2.0 * p.cr[0], 2.0 * p.cr[1], 2.0 * p.cr[2],
                          p.ddd[0], p.ddd[1], p.ddd[2], p.aab[0], p.abb[0], p.aab[1], p.abb[1], p.aab[2], p.abb[2], p.xyz};
    int top = 64;
#pragma unroll
    for (int q = 0; q < 19; ++q) top = max(top, (__double2hiint(v[q]) >> 20) & 0x7FF);
#pragma unroll
    for (int q = 0; q < 19; ++q) C[q * st] = __longlong_as_double(to_fixed<6>(bits_of(v[q]), top));
    C[19 * st] = __longlong_as_double(top);
}

// Twice the derivative along axis B (times h) of the R4 polynomial on the face x_D = NS/2, at the 2x2 Gauss points:
// the gradient of evaluate_grad (Navier-Stokes-3D/reconstruction.c:24-35) is bilinear there,
// P + Q t1 + R t2 + S t1 t2, with the squares t1^2 = t2^2 = 1/12 and |t1| = |t2| = GPT folded in.  Integers, in the
// coefficients' units: the 22 forms of a face at its four points were 340 of its 810 FP64 operations.
template <int D, int NS, int B>
__device__ __forceinline__ void face_form64(const double* __restrict__ C, long long st, i64& P, i64& Q, i64& R, i64& S) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    constexpr i64 kG2 = 2662558164157085696ll, kG8 = 665639541039271424ll;                // 2^64 times GPT/2 and GPT/8
    constexpr i64 k6 = 3074457345618258603ll, k12 = 1537228672809129301ll, k48 = 384307168202282325ll;  // 1/6, 1/12, 1/48
    auto ld = [&](int q) { return (i64)__double_as_longlong(__ldg(C + q * st)); };
    auto lin = [&](int a) { return ld(a); };
    auto sq = [&](int a) { return ld(3 + a); };
    auto cr2 = [&](int a, int b) { return ld(6 + pair_of(a, b)); };
    auto cube = [&](int a) { return ld(9 + a); };
    auto sqlin = [&](int a, int b) { return ld((a < b ? 12 : 13) + 2 * pair_of(a, b)); };  // of x_a^2 x_b
    auto toward = [&](i64 a, i64 b) { return NS > 0 ? a + b : a - b; };
    if constexpr (B == D) {
        P = toward(lin(D), sq(D)) - scaled(cube(D), split(k12));
        Q = scaled(toward(cr2(D, T1), sqlin(D, T1)), split(kG2));
        R = scaled(toward(cr2(D, T2), sqlin(D, T2)), split(kG2));
        S = scaled(ld(18), split(k48));
    } else {
        constexpr int O = B == T1 ? T2 : T1;
        P = toward(lin(B) - scaled(cube(B), split(k6)) + scaled(sqlin(D, B), split(k12)), (cr2(D, B) + 2) >> 2);
        // 2 GPT sq +- GPT/2 sqlin, GPT/2 cr2 +- GPT/8 xyz
        const i64 q = toward(4 * scaled(sq(B), split(kG2)), scaled(sqlin(B, D), split(kG2)));
        const i64 r = toward(scaled(cr2(B, O), split(kG2)), scaled(ld(18), split(kG8)));
        Q = B == T1 ? q : r;
        R = B == T1 ? r : q;
        S = scaled(sqlin(B, O), split(k12));
    }
}

// form k of a side, in the order visc_point64 takes them: rho along D, T1, T2; m_D likewise; m_T1 along D and T1;
// m_T2 along D and T2; E along D
constexpr int NFORM = 11;
template <int D, int NS, int K>
__device__ __forceinline__ void side_form64(const double* __restrict__ C4, long long NE, i64& P, i64& Q, i64& R, i64& S) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    constexpr int var = K < 3 ? 0 : K < 6 ? 1 + D : K < 8 ? 1 + T1 : K < 10 ? 1 + T2 : 4;
    constexpr int along = K == 1 || K == 4 || K == 7 ? T1 : K == 2 || K == 5 || K == 9 ? T2 : D;
    face_form64<D, NS, along>(C4 + var * 20 * NE, NE, P, Q, R, S);
}

// The viscous fluxes (PDEViscFlux, Navier-Stokes-3D/pde.c:90-162) of one face side at Gauss point gp, divided by
// mu/(2 h): Newtonian stress with Stokes' hypothesis and Fourier heat flux, with the program's velocity
// gradients u_x = (rho u)_x - u rho_x / rho (:118-130).  Adds the momentum components along D, T1, T2 and the
// energy's to av; Q is the side's trace, grad(k) the value of its form k, kmu = k / mu; returns 1 / rho.  Only the
// 11 gradient components that enter the flux along D are formed.
template <int D, class Grad>
__device__ __forceinline__ double visc_point64(const double* __restrict__ Q, Grad grad, double gm1, double kmu, double* av) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    const double rho = Q[0], md = Q[1 + D], m1 = Q[1 + T1], m2 = Q[1 + T2], E = Q[4];
    const double ir = recip_fix(rho);
    const double u = md * ir, v = m1 * ir, w = m2 * ir;
    const double em = fma(-w, m2, fma(-v, m1, fma(-u, md, E)));  // E - |m|^2 / rho
    const double rd = grad(0) * ir, r1 = grad(1) * ir, r2 = grad(2) * ir;
    const double gd = grad(3), g1 = grad(6), g2 = grad(8);
    const double ud = fma(-u, rd, gd), u1 = fma(-u, r1, grad(4)), u2 = fma(-u, r2, grad(5));
    const double vd = fma(-v, rd, g1), v1 = fma(-v, r1, grad(7));
    const double wd = fma(-w, rd, g2), w2 = fma(-w, r2, grad(9));
    // the temperature gradient (times c_v) of pde.c:118-130, regrouped:
    // (gamma - 1)/rho (E_D - u.m_D - rho_D/rho (E - |m|^2 / rho))
    const double um = fma(w, g2, fma(v, g1, u * gd));
    const double td = fma(-rd, em, grad(10) - um) * (gm1 * ir);
    const double tn = fma(-2. / 3., (ud + v1) + w2, 2.0 * ud), t1 = u1 + vd, t2 = u2 + wd;
    av[0] += tn;
    av[1] += t1;
    av[2] += t2;
    av[3] += fma(kmu, td, fma(w, t2, fma(v, t1, u * tn)));
    return ir;
}

}  // namespace euler
}  // namespace hype
