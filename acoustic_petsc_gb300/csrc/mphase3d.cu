// mphase3d.cu -- the 3D primitive-variable multiphase path of HyPE
// (3d/weno4/Viscous-Multiphase-Fourth-Order, RHSFunctionPrimitive, rhs_function.c:56-570):
// Q = (rho, rho u, rho v, rho w, E, phi) with the mixture EOS of two stiffened gases
// mixed by phi (pde.c:9-45), CWENO4 of the primitive variables, the 33-node
// admissibility check of PDECheckPAD with first order on failure (:284-306), the
// rotated HLLC flux with the normal velocity as a 7th component (pde.c:273-440), the
// non-conservative phi equation d phi/dt = -div(phi u) + phi div u (:507-552), and
// dt = (1/3) CFL h / (s_max + 2 s_visc / h) (:559), s_visc the viscous speed
// (4/3)(phi mu1 + (1 - phi) mu2)/rho of PDEViscFluxPrim (pde.c:101-136).  The program's
// viscous flux itself reads gradients that its weno() never writes; with zero gradients it
// is a signed zero, so no viscous flux is applied here.
//
// Per RHS evaluation:
//   k_m3_ghost   conservative SoA -> primitive with 3 ghost layers (boundary maps per
//                axis: periodic, transmissive copy, reflective mirror with the normal
//                velocity negated, rhs_function.c:98-230);
//   k_m3_recon   per extended cell and variable: CWENO4, the 24 face traces, and the 33-node check of
//                density and pressure (a bound on the polynomial first, node values where it fails);
//   k_m3_first_order  the cell values as traces where a node failed;
//   k_m3_faces   per face and Gauss point: the rotated HLLC flux (7 components), wave-speed maxima;
//   k_m3_update  RHS with the phi term, fused with the SSP stage combination.
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "cweno_fix.cuh"

namespace hype {
namespace mp3d {

using euler::NTR;
using euler::S1;
using euler::SO;
using euler::SQ;

constexpr int MV = 6;  // variables
constexpr int MF = 7;  // flux components (6 + the normal velocity of the phi term)
constexpr int GW = 3;
constexpr double RHO_FLOOR = 1.0e-14, PRS_FLOOR = 1.0e-12;

struct Geo {
    int nx, ny, nz;
    int bc[6];
    long long N, NE, GN;
    int ex, ey, gx, gy;
};

struct Eos {
    double g1, p1, g2, p2, mu1, mu2;
    // formed once on the host: g1 - 1, g2 - g1, (g1 - 1)(g2 - 1) and its reciprocal, and g p / (g - 1) of
    // the second gas and of the difference first - second
    double g1m, dg, k, rk, c2, dc;
    int stiff;
};

inline Eos make_eos(double g1, double p1, double g2, double p2, double mu1, double mu2) {
    const double c1 = g1 * p1 / (g1 - 1.0), c2 = g2 * p2 / (g2 - 1.0), k = (g1 - 1.0) * (g2 - 1.0);
    return Eos{g1, p1, g2, p2, mu1, mu2, g1 - 1.0, g2 - g1, k, 1.0 / k, c2, c1 - c2, p1 != 0.0 || p2 != 0.0};
}

struct DevScalars {
    unsigned long long smax_bits[6];   // [0..3] stages, [4] RHS-only calls
    unsigned long long smaxv_bits[6];  // viscous speeds, same slots
    double dt, t;
    unsigned long long bad;            // first inadmissible face's cell (ULLONG_MAX: none)
    unsigned long long fallback;       // owned-cell first-order fallbacks
};

// ---------------------------------------------------------------- EOS (pde.c:9-45)
// With d = (1 - phi)(g1 - 1) + phi (g2 - 1), linear in phi, and k = (g1 - 1)(g2 - 1):
//   gamma - 1 = k / d, 1 / (gamma - 1) = d / k, and gamma P_inf / (gamma - 1) = c1 phi + c2 (1 - phi), c = g p / (g - 1),
// so a state costs one reciprocal.
__device__ __forceinline__ double mix_d(const Eos& e, double phi) { return fma(phi, e.dg, e.g1m); }
__device__ __forceinline__ double mix_c(const Eos& e, double phi) { return fma(phi, e.dc, e.c2); }
// P_inf = (gamma - 1) / gamma (c1 phi + c2 (1 - phi)), 0 with no stiffness in either gas
__device__ __forceinline__ double mix_pinf(const Eos& e, double phi) {
    return e.stiff ? e.k / (mix_d(e, phi) + e.k) * mix_c(e, phi) : 0.0;
}
__device__ __forceinline__ void cons2prim(const Eos& e, const double* Q, double* V) {
    const double gm1 = e.k * euler::recip_fix(mix_d(e, Q[5]));
    const double ir = euler::recip_fix(Q[0]);
    double pe = fma(-0.5 * ir, fma(Q[3], Q[3], fma(Q[2], Q[2], Q[1] * Q[1])), Q[4]);
    if (e.stiff) pe -= mix_c(e, Q[5]);
    V[0] = Q[0];
    V[1] = Q[1] * ir;
    V[2] = Q[2] * ir;
    V[3] = Q[3] * ir;
    V[4] = gm1 * pe;
    V[5] = Q[5];
}

// One side of a Gauss point: the primitive trace, E + p and the sound speed (PDEConsFluxPrim, PDEPrim2Cons:
// pde.c:142-202, 27-45)
struct Side {
    double rho, u, v, w, p, phi, H, a;
};

// x < c for a positive c as the floating comparison decides it (false for NaN), on the bit pattern
__device__ __forceinline__ bool below(double x, double c) {
    const long long b = __double_as_longlong(x);
    return b < __double_as_longlong(c) && (unsigned long long)b <= 0xFFF0000000000000ull;
}
// x / 2, x zero, normal or not finite
__device__ __forceinline__ double half_of(double x) {
    const int hi = __double2hiint(x);
    return ((unsigned)(hi >> 20) & 0x7FFu) - 2u < 2045u ? __hiloint2double(hi - (1 << 20), __double2loint(x)) : x;
}

__device__ __forceinline__ Side make_side(const Eos& e, const double* V, bool& bad) {
    Side s;
    s.rho = V[0]; s.u = V[1]; s.v = V[2]; s.w = V[3]; s.p = V[4]; s.phi = V[5];
    const double d = mix_d(e, s.phi);
    const double gm1 = e.k * euler::recip_fix(d);
    double gp = fma(gm1, s.p, s.p);                  // gamma (p + P_inf)
    double pe = fma(d * e.rk, s.p, s.p);             // p + (p + gamma P_inf) / (gamma - 1)
    if (e.stiff) {
        const double c = mix_c(e, s.phi);
        gp = fma(gm1, c, gp);
        pe += c;
        bad |= below(gp, PRS_FLOOR * (1.0 + gm1));
    } else {
        bad |= below(s.p, PRS_FLOOR);
    }
    bad |= below(s.rho, RHO_FLOOR);
    s.H = fma(half_of(s.rho), fma(s.w, s.w, fma(s.v, s.v, s.u * s.u)), pe);
    s.a = euler::sqrt_fix(gp * euler::recip_fix(s.rho));
    return s;
}

// comparisons of a number with zero as the floating ones decide them (false for NaN), on the bit pattern
__device__ __forceinline__ bool above0(double x) {
    const long long b = __double_as_longlong(x);
    return b > 0 && b <= 0x7FF0000000000000ll;
}
__device__ __forceinline__ bool below0(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return b > 0x8000000000000000ull && b <= 0xFFF0000000000000ull;
}
__device__ __forceinline__ bool from0(double x) {  // x >= 0
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return b <= 0x7FF0000000000000ull || b == 0x8000000000000000ull;
}
__device__ __forceinline__ bool abs_above(double x, double y) {  // |x| > |y|, neither NaN
    return (__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll) > (__double_as_longlong(y) & 0x7FFFFFFFFFFFFFFFll);
}
__device__ __forceinline__ double neg_if(bool c, double x) {
    return __hiloint2double(__double2hiint(x) ^ (c ? 0x80000000 : 0), __double2loint(x));
}

// What the three HLLC solves of a Gauss point add up to.  With un the normal velocity of the side K that the
// solve selects, e = S_star - un, z = e / (S - S_star) (so that the star state's density factor
// (S - un) / (S - S_star) is 1 + z) and Y = S e rho (1 + z), the flux of PDEHLLCRiemannSolver
// (pde.c:273-379) is, per component,
//   rho m, rho u m + p n + Y c, (E + p) m + Y S_star, phi m, m,     m = un + S z
// (z = Y = 0 outside the star region).  Everything that multiplies m depends on the side alone, so the
// solves' weighted m are summed per side and the components formed once.
struct HllcSum {
    double mL, mR, px, py, pz, en;
};

// The selection of pde.c:368-376 (0 left, 1 left star, 2 right star, 3 right): with S_L == 0 and
// S_star >= 0 the program leaves the flux unset, here zero (4)
__device__ __forceinline__ int hllc_select(double SL, double SR, double Ss) {
    return above0(SL) ? 0 : (from0(Ss) && below0(SL)) ? 1 : (below0(Ss) && from0(SR)) ? 2 : below0(SR) ? 3 : 4;
}

// The momentum of one solve along the unit normal n, weight wt: wt (p n + Y c).  The program builds the
// star velocity from (S_star, u.t1, u.t2) in its Miller-Colella frame M = [n; t1; t2] and the inverse of M
// (pde.c:290-323), which is u + e c with c the first column of M^-1.  Where |ny + nz| <= |ny - nz| the frame
// is orthonormal and c = n.  In the other branch its t2z (pde.c:302) differs from that of n x t1 by
// nz (ny - nz) il, and with q2 = (ny + nz)^2 + (nz - nx)^2 + (nx + ny)^2 = 1 / il^2 and d = nz (ny - nz),
// t1 x t2 / det = (q2 n + d (nz - nx, -(ny + nz), 0)) / (q2 + d (nx (nz - nx) - ny (ny + nz))).
// wp = wt p, wY = wt Y; sum, dif, b, q2: ny + nz, ny - nz, nz - nx and, where |sum| > |dif|, q2
__device__ __forceinline__ void hllc_momentum(double nx, double ny, double nz, double sum, double dif, double b, double q2,
                                              double wp, double wY, HllcSum& h) {
    double pn;
    if (abs_above(sum, dif)) {
        const double dz = nz * dif;
        const double Yr = wY * euler::recip_fix(fma(dz, fma(nx, b, -ny * sum), q2));
        pn = fma(q2, Yr, wp);
        const double g = dz * Yr;
        h.px = fma(g, b, h.px);
        h.py = fma(-g, sum, h.py);
    } else {
        pn = wp + wY;
    }
    h.px = fma(pn, nx, h.px);
    h.py = fma(pn, ny, h.py);
    h.pz = fma(pn, nz, h.pz);
}

// One solve of weight wt along a normal of any direction: adds to h, returns the wave speed
__device__ __forceinline__ double hllc_general(const Side& L, const Side& R, double nx, double ny, double nz, double sum,
                                               double dif, double b, double q2, double wt, HllcSum& h) {
    const double unL = fma(L.w, nz, fma(L.v, ny, L.u * nx)), unR = fma(R.w, nz, fma(R.v, ny, R.u * nx));
    const double SL = fmin(unR - R.a, unL - L.a), SR = fmax(unL + L.a, unR + R.a);
    const double rL = L.rho * (SL - unL), rR = R.rho * (SR - unR);
    const double Ss = fma(-rR, unR, fma(rL, unL, R.p - L.p)) * euler::recip_fix(rL - rR);
    const int sel = hllc_select(SL, SR, Ss);
    if (sel != 4) {
        const bool left = sel <= 1;
        const double un = left ? unL : unR, p = left ? L.p : R.p;
        double m = un, wY = 0.0;
        if (sel == 1 || sel == 2) {
            const double S = left ? SL : SR, e = Ss - un;
            const double z = e * euler::recip_fix(S - Ss);
            m = fma(S, z, un);
            wY = wt * ((S * e) * fma(left ? L.rho : R.rho, z, left ? L.rho : R.rho));
            h.en = fma(wY, Ss, h.en);
        }
        if (left) h.mL = fma(wt, m, h.mL);
        else h.mR = fma(wt, m, h.mR);
        hllc_momentum(nx, ny, nz, sum, dif, b, q2, wt * p, wY, h);
    }
    return euler::max_num(fabs(unL) + L.a, fabs(unR) + R.a);
}

// PDErotHLLCRiemannSolver (pde.c:383-440) across an axis face of normal D: HLLC along the velocity-jump
// direction n1 and its two Miller-Colella tangents, weighted by their projections on the face normal.  The
// tangents are perpendicular to the jump, so both sides have one normal velocity un there: the acoustic
// speeds are un -+ amax and S_star - un, and with it z and rho (1 + z), is the same for both tangents.
// Without a jump n1 is the face normal, the tangents' weights are exactly zero and only their wave
// speeds count.  About 210 FP64 operations (three general solves: about 800).
template <int D>
__device__ __forceinline__ double rot_hllc7(const Side& L, const Side& R, double* Flux) {
    const double du = R.u - L.u, dv = R.v - L.v, dw = R.w - L.w;
    const double dq2 = fma(dw, dw, fma(dv, dv, du * du));
    const bool still = below(dq2, 1.0E-20);  // |du| < 1e-10 (pde.c:391)
    double nx = D == 0 ? 1.0 : 0.0, ny = D == 1 ? 1.0 : 0.0, nz = D == 2 ? 1.0 : 0.0, a1 = 1.0;
    if (!still) {
        const double idq = euler::rsqrt_fix(dq2);
        const bool flip = __double2hiint(D == 0 ? du : D == 1 ? dv : dw) < 0;
        const double sg = neg_if(flip, idq);
        nx = du * sg; ny = dv * sg; nz = dw * sg;
        a1 = D == 0 ? nx : D == 1 ? ny : nz;
    }
    // t1 and t2 = n1 x t1 of pde.c:402-424
    const double sum = ny + nz, dif = ny - nz, b = nz - nx;
    const bool first = abs_above(sum, dif);
    double t1x = first ? sum : dif, t1y = b, t1z = first ? -(nx + ny) : nx - ny;
    const double q2 = fma(t1z, t1z, fma(t1y, t1y, t1x * t1x));
    const double il = euler::rsqrt_fix(q2);
    t1x *= il;
    t1y *= il;
    t1z *= il;
    double t2x = fma(ny, t1z, -nz * t1y), t2y = fma(nz, t1x, -nx * t1z), t2z = fma(nx, t1y, -ny * t1x);
    HllcSum h{0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double smax = hllc_general(L, R, nx, ny, nz, sum, dif, b, q2, a1, h);
    if (still) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const double tx = q ? t2x : t1x, ty = q ? t2y : t1y, tz = q ? t2z : t1z;
            const double unL = fma(L.w, tz, fma(L.v, ty, L.u * tx)), unR = fma(R.w, tz, fma(R.v, ty, R.u * tx));
            smax = euler::max_num(smax, euler::max_num(fabs(unL) + L.a, fabs(unR) + R.a));
        }
    } else {
        const double am = euler::max_pos(L.a, R.a);
        const double e = (L.p - R.p) * euler::recip_fix((L.rho + R.rho) * am);  // S_star - un
        const double zL = -e * euler::recip_fix(am + e), zR = e * euler::recip_fix(am - e);
        const double yL = e * fma(L.rho, zL, L.rho), yR = e * fma(R.rho, zR, R.rho);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            double tx = q ? t2x : t1x, ty = q ? t2y : t1y, tz = q ? t2z : t1z;
            double wt = D == 0 ? tx : D == 1 ? ty : tz;
            const bool flip = below0(wt);
            wt = neg_if(flip, wt);
            tx = neg_if(flip, tx); ty = neg_if(flip, ty); tz = neg_if(flip, tz);
            const double un = fma(L.w, tz, fma(L.v, ty, L.u * tx));
            const double SL = un - am, SR = un + am, Ss = un + e;
            const int sel = hllc_select(SL, SR, Ss);
            smax = euler::max_num(smax, fabs(un) + am);
            if (sel == 4) continue;
            const bool left = sel <= 1;
            double m = un, wY = 0.0;
            if (sel == 1 || sel == 2) {
                const double S = left ? SL : SR;
                m = fma(S, left ? zL : zR, un);
                wY = wt * (S * (left ? yL : yR));
                h.en = fma(wY, Ss, h.en);
            }
            if (left) h.mL = fma(wt, m, h.mL);
            else h.mR = fma(wt, m, h.mR);
            const double ts = ty + tz, tb = tz - tx, tf = tx + ty;
            hllc_momentum(tx, ty, tz, ts, ty - tz, tb, fma(tf, tf, fma(tb, tb, ts * ts)), wt * (left ? L.p : R.p), wY, h);
        }
    }
    const double qL = L.rho * h.mL, qR = R.rho * h.mR;
    Flux[0] = qL + qR;
    Flux[1] = fma(L.u, qL, fma(R.u, qR, h.px));
    Flux[2] = fma(L.v, qL, fma(R.v, qR, h.py));
    Flux[3] = fma(L.w, qL, fma(R.w, qR, h.pz));
    Flux[4] = fma(L.H, h.mL, fma(R.H, h.mR, h.en));
    Flux[5] = fma(L.phi, h.mL, R.phi * h.mR);
    Flux[6] = h.mL + h.mR;
    return smax;
}

// ---------------------------------------------------------------- admissibility nodes
// the 33 nodes of hype.h:93-96 (centre, 12 axis points, 8 corners, 12 edge midpoints)
__host__ __device__ constexpr double node(int m, int axis) {
    constexpr double X[33] = {0.0, 0.5, 0.25, -0.25, -0.5, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.5, 0.0, -0.5, 0.5,
                              0.0, -0.5, 0.5, 0.0, -0.5, 0.5, 0.0, -0.5, 0.5, -0.5, 0.5, -0.5, 0.5, -0.5, 0.5, -0.5};
    constexpr double Y[33] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.5, 0.25, -0.25, -0.5, 0.0, 0.0, 0.0, 0.0, 0.5, 0.5, 0.5, -0.5,
                              -0.5, -0.5, 0.5, 0.5, 0.5, -0.5, -0.5, -0.5, 0.0, 0.0, 0.0, 0.0, 0.5, 0.5, -0.5, -0.5};
    constexpr double Z[33] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.5, 0.25, -0.25, -0.5, 0.5, 0.5, 0.5, 0.5,
                              0.5, 0.5, -0.5, -0.5, -0.5, -0.5, -0.5, -0.5, 0.5, 0.5, -0.5, -0.5, 0.0, 0.0, 0.0, 0.0};
    return axis == 0 ? X[m] : axis == 1 ? Y[m] : Z[m];
}

// the basis monomials of evaluate_polynomial (reconstruction.c:12-21)
__host__ __device__ constexpr double mono(int k, double x, double y, double z) {
    constexpr double r1_12 = 1. / 12., r3_20 = 3. / 20.;
    switch (k) {
        case 0: return 1.0;
        case 1: return x;
        case 2: return y;
        case 3: return z;
        case 4: return x * x - r1_12;
        case 5: return y * y - r1_12;
        case 6: return z * z - r1_12;
        case 7: return x * y;
        case 8: return y * z;
        case 9: return z * x;
        case 10: return x * (x * x - r3_20);
        case 11: return y * (y * y - r3_20);
        case 12: return z * (z * z - r3_20);
        case 13: return (x * x - r1_12) * y;
        case 14: return x * (y * y - r1_12);
        case 15: return (y * y - r1_12) * z;
        case 16: return y * (z * z - r1_12);
        case 17: return (x * x - r1_12) * z;
        case 18: return x * (z * z - r1_12);
        default: return x * y * z;
    }
}

// the polynomial at node M, the terms whose monomial vanishes there left out
template <int M, int K = 0>
__device__ __forceinline__ double node_value(const double* c, double acc = 0.0) {
    if constexpr (K == 20) {
        return acc;
    } else {
        constexpr double w = mono(K, node(M, 0), node(M, 1), node(M, 2));
        if constexpr (w == 0.0) return node_value<M, K + 1>(c, acc);
        else return node_value<M, K + 1>(c, fma(c[K], w, acc));
    }
}

// true when some node has rho < floor
template <int M = 0>
__device__ __forceinline__ bool rho_fails(const double* c) {
    if constexpr (M == 33) {
        return false;
    } else {
        return (node_value<M>(c) < RHO_FLOOR) | rho_fails<M + 1>(c);
    }
}

// true when some node has p + P_inf(phi) < floor; phi's polynomial at ph[q * st] (read only with stiffness)
template <int M = 0>
__device__ __forceinline__ bool prs_fails(const double* cp, const double* ph, int st, const Eos& e) {
    if constexpr (M == 33) {
        return false;
    } else {
        double pinf = 0.0;
        if (e.stiff) {
            double cphi[20];
#pragma unroll
            for (int q = 0; q < 20; ++q) cphi[q] = ph[q * st];
            pinf = mix_pinf(e, node_value<M>(cphi));
        }
        return (node_value<M>(cp) + pinf < PRS_FLOOR) | prs_fails<M + 1>(cp, ph, st, e);
    }
}

// How far a polynomial can be from its cell value at any of the 33 nodes: the basis functions are at most
// 1/2 (linear), 1/6 (square), 1/4 (cross), 1/20 (cubic), 1/12 (mixed) and 1/8 there.
__device__ __forceinline__ double spread(const euler::Poly64& p) {
    const double l = (fabs(p.lin[0]) + fabs(p.lin[1])) + fabs(p.lin[2]);
    const double q = (fabs(p.sq[0]) + fabs(p.sq[1])) + fabs(p.sq[2]);
    const double x = (fabs(p.cr[0]) + fabs(p.cr[1])) + fabs(p.cr[2]);
    const double c = (fabs(p.ddd[0]) + fabs(p.ddd[1])) + fabs(p.ddd[2]);
    const double m = ((fabs(p.aab[0]) + fabs(p.abb[0])) + (fabs(p.aab[1]) + fabs(p.abb[1]))) + (fabs(p.aab[2]) + fabs(p.abb[2]));
    const double r = fma(1. / 64., fabs(p.xyz), fma(1. / 48., m, 0.05 * c));
    return fma(fabs(p.wr), r, fma(0.125, x, fma(1. / 12., q, 0.25 * l)));
}
// no node can be below a floor of 1e-12: 21 operations decide what 33 node values (300) would, except in
// cells near the floor; the margin 1e-9 covers the rounding of either
__device__ __forceinline__ bool surely_above(const euler::Poly64& p) {
    return fma(1.0 - 1.0e-9, p.u0, -spread(p)) > 2.0e-12;
}

// ---------------------------------------------------------------- kernels
__device__ __forceinline__ long long ghost_index(const Geo& g, int i, int j, int k) {
    return ((long long)(k + GW) * g.gy + (j + GW)) * g.gx + (i + GW);
}
__device__ __forceinline__ long long ext_index(const Geo& g, int i, int j, int k) {
    return ((long long)(k + 1) * g.ey + (j + 1)) * g.ex + (i + 1);
}

// The cells of every kernel are indexed flat: rows of 32 x-neighbours left a third of the lanes of a
// 42-wide box without a cell.
constexpr int kGhostThreads = 128, kReconThreads = 64, kUpdateThreads = 128;

struct Box3 {
    int i, j, k;
    __device__ __forceinline__ Box3(unsigned q, int nx, int ny) {
        const unsigned row = q / (unsigned)nx, pl = row / (unsigned)ny;
        i = (int)(q - row * (unsigned)nx);
        j = (int)(row - pl * (unsigned)ny);
        k = (int)pl;
    }
};

__global__ void __launch_bounds__(kGhostThreads) k_m3_ghost(const double* __restrict__ U, double* __restrict__ G, Geo g, Eos e) {
    const unsigned dst = blockIdx.x * (unsigned)kGhostThreads + threadIdx.x;
    if (dst >= (unsigned)g.GN) return;
    const Box3 b(dst, g.gx, g.gy);
    int fi = 0, fj = 0, fk = 0;
    const int mi = bmap(b.i - GW, g.nx, g.bc[0], g.bc[1], &fi);
    const int mj = bmap(b.j - GW, g.ny, g.bc[2], g.bc[3], &fj);
    const int mk = bmap(b.k - GW, g.nz, g.bc[4], g.bc[5], &fk);
    const long long src = ((long long)mk * g.ny + mj) * g.nx + mi;
    double Q[MV], V[MV];
#pragma unroll
    for (int c = 0; c < MV; ++c) Q[c] = __ldg(U + c * g.N + src);
    cons2prim(e, Q, V);
    if (fi) V[1] = -V[1];
    if (fj) V[2] = -V[2];
    if (fk) V[3] = -V[3];
#pragma unroll
    for (int c = 0; c < MV; ++c) G[c * g.GN + dst] = V[c];
}

__device__ __forceinline__ void gather33(const double* __restrict__ p, int sy, int sz, double* s) {
    s[0] = __ldg(p);
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        const int off = (o == 0) ? -2 : (o == 1) ? -1 : (o == 2) ? 1 : 2;
        s[S1(0, off)] = __ldg(p + off);
        s[S1(1, off)] = __ldg(p + off * sy);
        s[S1(2, off)] = __ldg(p + off * sz);
    }
#pragma unroll
    for (int sa = 0; sa < 2; ++sa)
#pragma unroll
        for (int sb = 0; sb < 2; ++sb) {
            s[SQ(0, sa, 1, sb)] = __ldg(p + (2 * sa - 1) + (2 * sb - 1) * sy);
            s[SQ(1, sa, 2, sb)] = __ldg(p + (2 * sa - 1) * sy + (2 * sb - 1) * sz);
            s[SQ(0, sa, 2, sb)] = __ldg(p + (2 * sa - 1) + (2 * sb - 1) * sz);
        }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int d = 0; d < 2; ++d) s[SO(a, b, d)] = __ldg(p + (2 * a - 1) + (2 * b - 1) * sy + (2 * d - 1) * sz);
}

// T[c][face*4+gp][extended cell]; the cells the faces of owned cells need (at most one coordinate outside
// the grid).  One thread per cell and variable (blockIdx.y), as the single-gas reconstruction: a cell's six
// variables in turn left a 40 x 40 x 100 grid less than four waves of 2300-instruction threads.  Density and
// pressure are checked at the nodes; with stiffness the pressure check needs phi's polynomial, so that thread
// does phi first (blockIdx.y = 4: phi and p).  A failing cell is marked and its traces replaced by
// k_m3_first_order, since its variables are in different threads.
// Bound: integer issue, as the single-gas reconstruction (cweno_fix.cuh).
// The FP64 form of a variable that no check needs, with the stencil gathered again, so that the integer form's
// registers do not hold it (inlined: a 40 x 40 x 100 run of two steps 8.37 -> 8.86 ms)
static __device__ __noinline__ void m3_general(const double* __restrict__ p, int sy, int sz, double* __restrict__ T, long long NE) {
    double s[33];
    gather33(p, sy, sz, s);
    euler::Poly64 poly;
    euler::cweno4_64(s, poly);
    euler::store_traces64(poly, T, NE);
}

__global__ void __launch_bounds__(kReconThreads, 5) k_m3_recon(const double* __restrict__ G, double* __restrict__ T, Geo g, Eos e,
                                                            unsigned char* __restrict__ fail) {
    __shared__ double sphi[20 * kReconThreads];  // phi's coefficients, [q][thread]
    const unsigned e_ = blockIdx.x * (unsigned)kReconThreads + threadIdx.x;
    if (e_ >= (unsigned)g.NE) return;
    const Box3 b(e_, g.ex, g.ey);
    const int i = b.i - 1, j = b.j - 1, k = b.k - 1;
    const int outside = (i < 0 || i >= g.nx) + (j < 0 || j >= g.ny) + (k < 0 || k >= g.nz);
    if (outside > 1) return;
    const long long ge = ghost_index(g, i, j, k);
    const int sy = g.gx, sz = g.gx * g.gy;
    double* ph = sphi + threadIdx.x;
    const int last = blockIdx.y;  // 0..3, then p; without stiffness phi is a sixth row of blocks
    bool phi_above = true;
#pragma unroll 1
    for (int c = (e.stiff && last == 4) ? 5 : last;; c = last) {
        const bool check = c == 0 || c == 4;
        double s[33];
        gather33(G + c * g.GN + ge, sy, sz, s);
        double* Tc = T + (long long)c * NTR * g.NE + e_;
        euler::PolyFix fix;
        const bool fixed = euler::recon_fix<false>(s, check, Tc, g.NE, fix);
        if (!fixed && !check && c == last) {
            m3_general(G + c * g.GN + ge, sy, sz, Tc, g.NE);
            break;
        }
        bool fp64 = !fixed;  // whether the FP64 polynomial is needed
        if (fixed) {
            if (c != last) {  // phi: P_inf >= 0 wherever 0 <= phi <= 1
                const double u = euler::from_fixed(fix.u0, fix.top), sp = euler::from_fixed((long long)euler::spread_fix(fix), fix.top);
                fp64 = !(phi_above = u - sp >= 0.0 && u + sp <= 1.0 && e.p1 >= 0.0 && e.p2 >= 0.0);
            } else if (check) {
                fp64 = !(phi_above && euler::surely_above(fix, 2.0e-12));
            }
        }
        if (fp64) {
            euler::Poly64 poly;
            euler::cweno4_64(s, poly);
            if (!fixed) euler::store_traces64(poly, Tc, g.NE);
            if (c != last) {
                const double sp = spread(poly);
                phi_above = poly.u0 - sp >= 0.0 && poly.u0 + sp <= 1.0 && e.p1 >= 0.0 && e.p2 >= 0.0;
            }
            if (c != last || (check && !(phi_above && surely_above(poly)))) {
                double cf[20];
                euler::coeffs64(poly, cf);
                if (c != last) {
#pragma unroll
                    for (int q = 0; q < 20; ++q) ph[q * kReconThreads] = cf[q];
                } else {
                    if (e.stiff && c == 4 && phi_above) {  // phi's polynomial was not kept: form it again
                        double sf[33], cp[20];
                        gather33(G + 5 * g.GN + ge, sy, sz, sf);
                        euler::cweno4_64(sf, poly);
                        euler::coeffs64(poly, cp);
#pragma unroll
                        for (int q = 0; q < 20; ++q) ph[q * kReconThreads] = cp[q];
                    }
                    if (c == 0 ? rho_fails(cf) : prs_fails(cf, ph, kReconThreads, e)) fail[e_] = 1;
                }
            }
        }
        if (c == last) break;
    }
}

// first order where a node was inadmissible: every trace is the cell value (rhs_function.c:302-306)
__global__ void __launch_bounds__(128) k_m3_first_order(const double* __restrict__ G, double* __restrict__ T, Geo g,
                                                        unsigned char* __restrict__ fail, DevScalars* __restrict__ ds) {
    const unsigned e_ = blockIdx.x * 128u + threadIdx.x;
    if (e_ >= (unsigned)g.NE || !fail[e_]) return;
    fail[e_] = 0;
    const Box3 b(e_, g.ex, g.ey);
    const int i = b.i - 1, j = b.j - 1, k = b.k - 1;
    const long long ge = ghost_index(g, i, j, k);
#pragma unroll 1
    for (int c = 0; c < MV; ++c) {
        const double v = G[c * g.GN + ge];
#pragma unroll
        for (int q = 0; q < NTR; ++q) T[((long long)c * NTR + q) * g.NE + e_] = v;
    }
    if (i >= 0 && i < g.nx && j >= 0 && j < g.ny && k >= 0 && k < g.nz) atomicAdd(&ds->fallback, 1ull);
}

// The maximum only grows while a kernel runs: a warp that does not exceed what it reads leaves it alone
__device__ __forceinline__ void raise_max(unsigned long long* a, double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (v > 0.0 && b > *(volatile unsigned long long*)a) atomicMax(a, b);
}

// Faces normal to D: the low cell's face 2D+1 against the high cell's face 2D.  All three directions in one
// launch (blockIdx.y); a block is 32 faces, indexed flat, x the 4 Gauss points, one point per warp, summed
// through shared memory.  Bound: FP64 issue.  With one thread per face, its four points in turn, and three
// general solves per point the three face launches of a 40 x 40 x 100 RHS took 3.9 ms of 5.6; a whole RHS
// and stage then took 1.9 ms (22.5 -> 7.5 ms per step); with reciprocals and roots on the integer pipe the
// faces are 0.77 ms (4.1 ms per step).
template <int D>
__device__ __forceinline__ void faces(const double* __restrict__ T, double* __restrict__ F, const Geo& g, const Eos& e,
                                      DevScalars* __restrict__ ds, int slot, double (*sh)[MF][32]) {
    const int lane = threadIdx.x & 31, gp = threadIdx.x >> 5;
    const unsigned f = blockIdx.x * 32u + lane;
    const unsigned fx = g.nx + (D == 0), fy = g.ny + (D == 1), nf = fx * fy * (g.nz + (D == 2));
    if (blockIdx.x * 32u >= nf) return;  // the grid is as wide as the direction with the most faces
    double smax = 0.0, smaxv = 0.0;
    if (f < nf) {
        const Box3 b(f, (int)fx, (int)fy);
        const double* TL = T + ((2 * D + 1) * 4 + gp) * g.NE + ext_index(g, b.i - (D == 0), b.j - (D == 1), b.k - (D == 2));
        const double* TR = T + (2 * D * 4 + gp) * g.NE + ext_index(g, b.i, b.j, b.k);
        double VL[MV], VR[MV], fc[MF];
#pragma unroll
        for (int c = 0; c < MV; ++c) {
            VL[c] = __ldg(TL + c * NTR * g.NE);
            VR[c] = __ldg(TR + c * NTR * g.NE);
        }
        bool bad = false;
        const Side SL = make_side(e, VL, bad), SR = make_side(e, VR, bad);
        smax = rot_hllc7<D>(SL, SR, fc);
        if (e.mu1 != 0.0 || e.mu2 != 0.0) {  // PDEViscFluxPrim's speed (4/3) mu / rho on both sides
            const double r4_3 = 4. / 3;
            const double svl = r4_3 * (VL[5] * e.mu1 + (1.0 - VL[5]) * e.mu2) / VL[0];
            const double svr = r4_3 * (VR[5] * e.mu1 + (1.0 - VR[5]) * e.mu2) / VR[0];
            smaxv = fmax(0.0, fmax(svl, svr));
        }
#pragma unroll
        for (int c = 0; c < MF; ++c) sh[gp][c][lane] = fc[c];
        if (bad) {
            const int ci = min(b.i, g.nx - 1), cj = min(b.j, g.ny - 1), ck = min(b.k, g.nz - 1);
            atomicMin(&ds->bad, (unsigned long long)(((long long)ck * g.ny + cj) * g.nx + ci));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        smax = euler::max_num(smax, __shfl_xor_sync(0xffffffffu, smax, o));
        smaxv = euler::max_num(smaxv, __shfl_xor_sync(0xffffffffu, smaxv, o));
    }
    if (lane == 0) {
        raise_max(&ds->smax_bits[slot], smax);
        raise_max(&ds->smaxv_bits[slot], smaxv);
    }
    __syncthreads();
    for (int c = gp; c < MF; c += 4)
        if (f < nf)
            F[(long long)c * nf + f] = euler::sum4(sh[0][c][lane], sh[1][c][lane], sh[2][c][lane], sh[3][c][lane], 2);
}

__global__ void __launch_bounds__(128) k_m3_faces(const double* __restrict__ T, double* __restrict__ Fx, double* __restrict__ Fy,
                                                  double* __restrict__ Fz, Geo g, Eos e, DevScalars* __restrict__ ds, int slot) {
    __shared__ double sh[4][MF][32];
    if (blockIdx.y == 0) faces<0>(T, Fx, g, e, ds, slot, sh);
    else if (blockIdx.y == 1) faces<1>(T, Fy, g, e, ds, slot, sh);
    else faces<2>(T, Fz, g, e, ds, slot, sh);
}

struct Stage {
    double a, b, c;  // out = a U + b W + (c dt) L (a = 0: W + (c dt) L); rhs_only: out = L
    int rhs_only;
};

// RHS (rhs_function.c:507-552) and the stage combination; Win: the stage input, whose
// volume fraction multiplies the normal-velocity flux in the phi equation
// Win, U, W and out may be one array (in-place stages), so they carry no __restrict__
__global__ void __launch_bounds__(kUpdateThreads) k_m3_update(const double* __restrict__ Fx, const double* __restrict__ Fy,
                                                              const double* __restrict__ Fz, const double* Win,
                                                              const double* U, const double* W,
                                                              double* out, Geo g, double r1_h, Stage st,
                                                              const DevScalars* __restrict__ ds) {
    const unsigned cell = blockIdx.x * (unsigned)kUpdateThreads + threadIdx.x;
    if (cell >= (unsigned)g.N) return;
    const unsigned row = cell / (unsigned)g.nx, k = row / (unsigned)g.ny;
    const int c = blockIdx.y;
    const long long nfx = (long long)(g.nx + 1) * g.ny * g.nz, nfy = (long long)g.nx * (g.ny + 1) * g.nz,
                    nfz = (long long)g.nx * g.ny * (g.nz + 1);
    const long long ix = cell + row, iy = cell + k * (unsigned)g.nx, iz = cell, sxy = (long long)g.nx * g.ny;
    const double cdt = st.rhs_only ? 0.0 : st.c * ds->dt;
    // the flux difference of component q over the three directions
    auto div = [&](int q) {
        return euler::sum_differences(Fx[q * nfx + ix + 1], Fx[q * nfx + ix], Fy[q * nfy + iy + g.nx], Fy[q * nfy + iy],
                                      Fz[q * nfz + iz + sxy], Fz[q * nfz + iz]);
    };
    double L = div(c);
    if (c == 5) L = fma(-Win[5 * g.N + cell], div(6), L);
    L *= -r1_h;
    double v = L;
    if (!st.rhs_only) {
        v = W[c * g.N + cell] + cdt * L;
        if (st.a != 0.0) v = st.a * U[c * g.N + cell] + st.b * W[c * g.N + cell] + cdt * L;
    }
    out[c * g.N + cell] = v;
}

// dt = (1/3) CFL h / (s_max + 2 s_visc / h) (rhs_function.c:559)
__host__ __device__ inline double m3_dt(double cfl_h, double r1_h, double smax, double smaxv) {
    return (1.0 / 3.0) * cfl_h / (smax + (r1_h * smaxv) * 2.0);
}

__global__ void k_m3_begin(DevScalars* ds, int dt_mode, int src, int use_src, int reset, double cfl_h, double r1_h) {
    if (use_src && dt_mode != HYPE_DT_FIXED) {
        ds->dt = m3_dt(cfl_h, r1_h, __longlong_as_double((long long)ds->smax_bits[src]),
                       __longlong_as_double((long long)ds->smaxv_bits[src]));
    }
    if (reset)
        for (int s = 0; s < 4; ++s) ds->smax_bits[s] = ds->smaxv_bits[s] = 0ull;
    ds->t += ds->dt;
}

__global__ void k_m3_reset_slot(DevScalars* ds, int slot) {
    ds->smax_bits[slot] = 0ull;
    ds->smaxv_bits[slot] = 0ull;
    ds->bad = ~0ull;
}

__global__ void k_m3_aos2soa(const double* __restrict__ a, double* __restrict__ s, long long N) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= N * MV) return;
    const long long cell = q / MV;
    s[(q - cell * MV) * N + cell] = a[q];
}
__global__ void k_m3_soa2aos(const double* __restrict__ s, double* __restrict__ a, long long N) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= N * MV) return;
    const long long cell = q / MV;
    a[q] = s[(q - cell * MV) * N + cell];
}

}  // namespace mp3d
}  // namespace hype

using namespace hype;
using namespace hype::mp3d;

static inline double bits2d3(unsigned long long b) {
    double d;
    memcpy(&d, &b, sizeof(d));
    return d;
}

struct hype_mp3d {
    hype_mp3d_params p;
    Geo g;
    Eos e;
    cudaStream_t stream = nullptr;
    double *U = nullptr, *W = nullptr, *S = nullptr, *L = nullptr, *G = nullptr, *T = nullptr;
    double *Fx = nullptr, *Fy = nullptr, *Fz = nullptr, *aos = nullptr;
    unsigned char* fail = nullptr;  // per extended cell: first order in this RHS; zero between RHS calls
    DevScalars* ds = nullptr;
    DevScalars* hs = nullptr;
};

static int m3_rhs(hype_mp3d* m, const double* Win, int slot) {
    const Geo& g = m->g;
    k_m3_ghost<<<cdiv(g.GN, kGhostThreads), kGhostThreads, 0, m->stream>>>(Win, m->G, g, m->e);
    k_m3_recon<<<dim3(cdiv(g.NE, kReconThreads), m->e.stiff ? 5 : 6), kReconThreads, 0, m->stream>>>(m->G, m->T, g, m->e, m->fail);
    k_m3_first_order<<<cdiv(g.NE, 128), 128, 0, m->stream>>>(m->G, m->T, g, m->fail, m->ds);
    const long long most = std::max({(long long)(g.nx + 1) * g.ny * g.nz, (long long)g.nx * (g.ny + 1) * g.nz,
                                     (long long)g.nx * g.ny * (g.nz + 1)});
    k_m3_faces<<<dim3(cdiv(most, 32), 3), 128, 0, m->stream>>>(m->T, m->Fx, m->Fy, m->Fz, g, m->e, m->ds, slot);
    HYPE_LAUNCHED(4);
    return HYPE_OK;
}

static int m3_update(hype_mp3d* m, const double* Win, const double* U, const double* W, double* out, Stage st) {
    const Geo& g = m->g;
    k_m3_update<<<dim3(cdiv(g.N, kUpdateThreads), MV), kUpdateThreads, 0, m->stream>>>(
        m->Fx, m->Fy, m->Fz, Win, U, W, out, g, 1.0 / m->p.h, st, m->ds);
    HYPE_LAUNCHED(1);
    return HYPE_OK;
}

extern "C" int hype_mp3d_create(const hype_mp3d_params* p, hype_mp3d** out) {
    if (!p || !out) return HYPE_ERR_ARG;
    *out = nullptr;
    if (p->nx < 3 || p->ny < 3 || p->nz < 3 || !(p->h > 0) || !(p->cfl > 0)) return HYPE_ERR_ARG;
    for (int f = 0; f < 6; ++f)
        if (p->bc[f] < HYPE_BC_PERIODIC || p->bc[f] > HYPE_BC_TRANSMISSIVE) return HYPE_ERR_ARG;
    for (int d = 0; d < 3; ++d)
        if ((p->bc[2 * d] == HYPE_BC_PERIODIC) != (p->bc[2 * d + 1] == HYPE_BC_PERIODIC)) return HYPE_ERR_ARG;
    if (!(p->g1 > 1.0) || !(p->g2 > 1.0) || !(p->mu1 >= 0.0) || !(p->mu2 >= 0.0)) return HYPE_ERR_ARG;
    if (p->dt_mode < HYPE_DT_MONITOR || p->dt_mode > HYPE_DT_FIXED) return HYPE_ERR_ARG;
    hype_mp3d* m = new hype_mp3d();
    m->p = *p;
    m->e = make_eos(p->g1, p->p1, p->g2, p->p2, p->mu1, p->mu2);
    Geo& g = m->g;
    g.nx = p->nx; g.ny = p->ny; g.nz = p->nz;
    for (int f = 0; f < 6; ++f) g.bc[f] = p->bc[f];
    g.N = (long long)p->nx * p->ny * p->nz;
    g.ex = p->nx + 2; g.ey = p->ny + 2;
    g.NE = (long long)g.ex * g.ey * (p->nz + 2);
    g.gx = p->nx + 2 * GW; g.gy = p->ny + 2 * GW;
    g.GN = (long long)g.gx * g.gy * (p->nz + 2 * GW);
    const size_t sN = sizeof(double) * MV * (size_t)g.N;
    cudaError_t ce = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    auto al = [&](double** ptr, size_t bytes) {
        if (ce == cudaSuccess) ce = cudaMalloc((void**)ptr, bytes);
    };
    al(&m->U, sN); al(&m->W, sN); al(&m->S, sN); al(&m->L, sN); al(&m->aos, sN);
    al(&m->G, sizeof(double) * MV * (size_t)g.GN);
    al(&m->T, sizeof(double) * MV * NTR * (size_t)g.NE);
    al(&m->Fx, sizeof(double) * MF * (size_t)(g.nx + 1) * g.ny * g.nz);
    al(&m->Fy, sizeof(double) * MF * (size_t)g.nx * (g.ny + 1) * g.nz);
    al(&m->Fz, sizeof(double) * MF * (size_t)g.nx * g.ny * (g.nz + 1));
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&m->fail, (size_t)g.NE);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(m->fail, 0, (size_t)g.NE, m->stream);
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&m->ds, sizeof(DevScalars));
    if (ce == cudaSuccess) ce = cudaMallocHost((void**)&m->hs, sizeof(DevScalars));
    if (ce == cudaSuccess) {
        DevScalars z;
        memset(&z, 0, sizeof(z));
        z.bad = ~0ull;
        ce = cudaMemcpy(m->ds, &z, sizeof(z), cudaMemcpyHostToDevice);
    }
    if (ce != cudaSuccess) {
        set_last_error("hype_mp3d_create", ce);
        hype_mp3d_destroy(m);
        return ce == cudaErrorMemoryAllocation ? HYPE_ERR_NOMEM : HYPE_ERR_CUDA;
    }
    *out = m;
    return HYPE_OK;
}

extern "C" void hype_mp3d_destroy(hype_mp3d* m) {
    if (!m) return;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->U); cudaFree(m->W); cudaFree(m->S); cudaFree(m->L); cudaFree(m->aos); cudaFree(m->G); cudaFree(m->T);
    cudaFree(m->Fx); cudaFree(m->Fy); cudaFree(m->Fz); cudaFree(m->fail); cudaFree(m->ds);
    if (m->hs) cudaFreeHost(m->hs);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

extern "C" int hype_mp3d_get_params(const hype_mp3d* m, hype_mp3d_params* out) {
    if (!m || !out) return HYPE_ERR_ARG;
    *out = m->p;
    return HYPE_OK;
}

static int m3_h2d(hype_mp3d* m, const double* aos, double* soa) {
    const long long N = m->g.N;
    HYPE_CK(cudaMemcpyAsync(m->aos, aos, sizeof(double) * MV * N, cudaMemcpyHostToDevice, m->stream));
    k_m3_aos2soa<<<cdiv(N * MV, 256), 256, 0, m->stream>>>(m->aos, soa, N);
    HYPE_LAUNCHED(1);
    return HYPE_OK;
}

static int m3_d2h(hype_mp3d* m, const double* soa, double* aos) {
    const long long N = m->g.N;
    k_m3_soa2aos<<<cdiv(N * MV, 256), 256, 0, m->stream>>>(soa, m->aos, N);
    HYPE_LAUNCHED(1);
    HYPE_CK(copy_to_host(aos, m->aos, sizeof(double) * MV * N, m->stream));
    HYPE_CK(cudaStreamSynchronize(m->stream));
    return HYPE_OK;
}

static int m3_scalars(hype_mp3d* m) {
    HYPE_CK(cudaMemcpyAsync(m->hs, m->ds, sizeof(DevScalars), cudaMemcpyDeviceToHost, m->stream));
    HYPE_CK(cudaStreamSynchronize(m->stream));
    return HYPE_OK;
}

extern "C" int hype_mp3d_upload(hype_mp3d* m, const double* U_aos) {
    if (!m || !U_aos) return HYPE_ERR_ARG;
    int rc = m3_h2d(m, U_aos, m->U);
    if (rc) return rc;
    HYPE_CK(cudaStreamSynchronize(m->stream));
    return HYPE_OK;
}

extern "C" int hype_mp3d_download(hype_mp3d* m, double* U_aos) {
    if (!m || !U_aos) return HYPE_ERR_ARG;
    return m3_d2h(m, m->U, U_aos);
}

extern "C" int hype_mp3d_rhs(hype_mp3d* m, double t, const double* U_aos, double* RHS_aos, double* dt_out) {
    (void)t;
    if (!m || !U_aos || !RHS_aos) return HYPE_ERR_ARG;
    int rc = m3_h2d(m, U_aos, m->S);
    if (rc) return rc;
    k_m3_reset_slot<<<1, 1, 0, m->stream>>>(m->ds, 4);
    HYPE_LAUNCHED(1);
    if ((rc = m3_rhs(m, m->S, 4)) || (rc = m3_update(m, m->S, nullptr, nullptr, m->L, Stage{0.0, 0.0, 0.0, 1})))
        return rc;
    if ((rc = m3_scalars(m))) return rc;
    if (dt_out)
        *dt_out = m3_dt(m->p.cfl * m->p.h, 1.0 / m->p.h, bits2d3(m->hs->smax_bits[4]), bits2d3(m->hs->smaxv_bits[4]));
    const bool bad = m->hs->bad != ~0ull;
    if ((rc = m3_d2h(m, m->L, RHS_aos))) return rc;
    return bad ? HYPE_ERR_STATE : HYPE_OK;
}

extern "C" int hype_mp3d_step(hype_mp3d* m, int nsteps, double* t_inout, double* dt_inout, long long* fallback_cells) {
    if (!m || nsteps < 0 || !t_inout || !dt_inout) return HYPE_ERR_ARG;
    const int mode = m->p.dt_mode;
    if (mode == HYPE_DT_FIXED && !(*dt_inout > 0)) return HYPE_ERR_ARG;
    const double cfl_h = m->p.cfl * m->p.h, r1_h = 1.0 / m->p.h;
    DevScalars init;
    memset(&init, 0, sizeof(init));
    init.t = *t_inout;
    init.dt = *dt_inout;
    init.bad = ~0ull;
    HYPE_CK(cudaMemcpyAsync(m->ds, &init, sizeof(init), cudaMemcpyHostToDevice, m->stream));
    const bool first_from_rhs = (mode != HYPE_DT_FIXED) && !(*dt_inout > 0);
    // SSPRK(4,3) (PETSc TSSSP RKS3, 4 stages, hype.c:207-209)
    const Stage s12{0.0, 1.0, 0.5, 0}, s3{2.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0, 0};
    int rc;
    for (int s = 0; s < nsteps; ++s) {
        if (s == 0 && first_from_rhs) {
            // the initial RHS call of hype.c:168 is this step's first stage RHS
            if ((rc = m3_rhs(m, m->U, 0))) return rc;
            k_m3_begin<<<1, 1, 0, m->stream>>>(m->ds, mode, 0, 1, 0, cfl_h, r1_h);
            HYPE_LAUNCHED(1);
        } else {
            k_m3_begin<<<1, 1, 0, m->stream>>>(m->ds, mode, 3, mode == HYPE_DT_MONITOR && s > 0, 1, cfl_h, r1_h);
            HYPE_LAUNCHED(1);
            if ((rc = m3_rhs(m, m->U, 0))) return rc;
        }
        if ((rc = m3_update(m, m->U, m->U, m->U, m->W, s12))) return rc;
        if ((rc = m3_rhs(m, m->W, 1)) || (rc = m3_update(m, m->W, m->U, m->W, m->W, s12))) return rc;
        if ((rc = m3_rhs(m, m->W, 2)) || (rc = m3_update(m, m->W, m->U, m->W, m->W, s3))) return rc;
        if ((rc = m3_rhs(m, m->W, 3)) || (rc = m3_update(m, m->W, m->U, m->W, m->U, s12))) return rc;
    }
    if ((rc = m3_scalars(m))) return rc;
    *t_inout = m->hs->t;
    *dt_inout = (nsteps > 0 && mode == HYPE_DT_MONITOR)
                    ? m3_dt(cfl_h, r1_h, bits2d3(m->hs->smax_bits[3]), bits2d3(m->hs->smaxv_bits[3]))
                    : m->hs->dt;
    if (fallback_cells) *fallback_cells = (long long)m->hs->fallback;
    return m->hs->bad == ~0ull ? HYPE_OK : HYPE_ERR_STATE;
}

extern "C" int hype_mp3d_sync(hype_mp3d* m) {
    if (!m) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(m->stream));
    return HYPE_OK;
}

extern "C" void* hype_mp3d_stream(hype_mp3d* m) { return m ? (void*)m->stream : nullptr; }
