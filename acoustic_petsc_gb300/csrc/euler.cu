// euler.cu -- 3D Euler CWENO4 + Rusanov RHS and the SSPRK(4,3) stepper on sm_103a.
//
// Per RK stage four kernels run on the context's stream (FP64; the other forms alike):
//   ghost  : the stage input with three ghost layers (replaces DMGlobalToLocal + the
//            BC sweeps of 3d/weno4/Navier-Stokes-3D/rhs_function.c:41-181);
//   recon  : one thread per variable and cell of the extended box [-1,n]^3 that some
//            face of an owned cell needs; writes the 24 face Gauss-point traces
//            (rhs_function.c:185-274);
//   faces  : all three directions; one Riemann solve per thread, the weighted flux
//            (rhs_function.c:276-417), the block max of the wave speed (atomicMax on
//            the bit pattern: speeds are >= 0) and the admissibility flag (replaces
//            MPI_Abort, pde.c:56-66);
//   update : flux divergence (rhs_function.c:419-433) fused with the SSP stage
//            combination; dt comes from device memory, so a whole step needs no
//            host round trip.
// State and stage buffers are SoA doubles [c][k][j][i]; traces are stored in the
// arithmetic type R of the reconstruction ([c][face][gp][extended cell]).
#include <cuda_runtime.h>

#include <string.h>

#include <algorithm>
#include <type_traits>

#include <vector>

#include "cweno_fix.cuh"
#include "euler_kernels.cuh"
#include "mlp_kernels.cuh"

namespace hype {
namespace euler {

struct Geo {
    int nx, ny, nz;
    int bc[6];
    long long N;   // owned cells
    long long NE;  // extended cells (n+2)^3
    int ex, ey;    // extended x, y extents
    int gx, gy;    // ghosted x, y extents (n + 2 GW): the stage input with its ghost layers
    long long GN;  // ghosted cells per variable
};

// ghost width of the stage-input copy: the reconstruction of the first ghost layer
// (i = -1) reads offsets down to -3
constexpr int GW = 3;

__host__ __device__ __forceinline__ void set_ghost_extents(Geo& g) {
    g.gx = g.nx + 2 * GW;
    g.gy = g.ny + 2 * GW;
    g.GN = (long long)g.gx * g.gy * (g.nz + 2 * GW);
}

__device__ __forceinline__ long long ghost_index(const Geo& g, int i, int j, int k) {
    return ((long long)(k + GW) * g.gy + (j + GW)) * g.gx + (i + GW);
}

// device scalars of one context
struct DevScalars {
    unsigned long long smax_bits[6];  // [0..3] stages, [4] RHS-only calls
    double dt;
    double t;
    unsigned long long bad;  // first inadmissible cell (ULLONG_MAX: none)
    long long rhs_evals;
    unsigned long long smaxv_bits[6];  // viscous wave speeds, same slots
};

// viscosity of the Navier-Stokes terms (mu = 0: Euler)
struct Visc {
    double mu, kc, vmax, r1_h;  // viscosity, cv mu gamma / Pr, max(4 mu / 3, gamma mu / Pr), 1 / h
};

__device__ __forceinline__ long long ext_index(const Geo& g, int i, int j, int k) {
    return ((long long)(k + 1) * (g.ny + 2) + (j + 1)) * (long long)g.ex + (i + 1);
}

// boundary maps of the offsets -2..2 of one cell along each direction
struct StencilMap {
    int mi[5], mj[5], mk[5];
    int fi, fj, fk;  // bit o set: offset o-2 is a reflective ghost
};

__device__ __forceinline__ void make_map(const Geo& g, int i, int j, int k, StencilMap& m) {
    m.fi = m.fj = m.fk = 0;
#pragma unroll
    for (int o = 0; o < 5; ++o) {
        int f = 0;
        m.mi[o] = bmap(i + o - 2, g.nx, g.bc[0], g.bc[1], &f);
        m.fi |= f << o;
        f = 0;
        m.mj[o] = bmap(j + o - 2, g.ny, g.bc[2], g.bc[3], &f);
        m.fj |= f << o;
        f = 0;
        m.mk[o] = bmap(k + o - 2, g.nz, g.bc[4], g.bc[5], &f);
        m.fk |= f << o;
    }
}

// one value of variable c at offset (oi, oj, ok) from the state (S = double) or its
// FP32 mirror (S = float); a reflective ghost negates the momentum component normal
// to its wall
template <typename R, typename S>
__device__ __forceinline__ R ldw(const S* __restrict__ Wc, int c, const Geo& g, const StencilMap& m, int oi, int oj,
                                 int ok) {
    S v = __ldg(Wc + ((long long)m.mk[ok + 2] * g.ny + m.mj[oj + 2]) * g.nx + m.mi[oi + 2]);
    const int fm = (c == 1) ? m.fi : (c == 2) ? m.fj : (c == 3) ? m.fk : 0;
    const int o = (c == 1) ? oi : (c == 2) ? oj : ok;
    if (fm && ((fm >> (o + 2)) & 1)) v = -v;
    return (R)v;
}

// the 33-point stencil of variable c (index map of euler_kernels.cuh)
template <typename R, typename S>
__device__ __forceinline__ void gather33(const S* __restrict__ Wc, int c, const Geo& g, const StencilMap& m, R* s) {
    s[0] = ldw<R>(Wc, c, g, m, 0, 0, 0);
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        const int off = (o == 0) ? -2 : (o == 1) ? -1 : (o == 2) ? 1 : 2;
        s[S1(0, off)] = ldw<R>(Wc, c, g, m, off, 0, 0);
        s[S1(1, off)] = ldw<R>(Wc, c, g, m, 0, off, 0);
        s[S1(2, off)] = ldw<R>(Wc, c, g, m, 0, 0, off);
    }
#pragma unroll
    for (int sa = 0; sa < 2; ++sa)
#pragma unroll
        for (int sb = 0; sb < 2; ++sb) {
            s[SQ(0, sa, 1, sb)] = ldw<R>(Wc, c, g, m, 2 * sa - 1, 2 * sb - 1, 0);
            s[SQ(1, sa, 2, sb)] = ldw<R>(Wc, c, g, m, 0, 2 * sa - 1, 2 * sb - 1);
            s[SQ(0, sa, 2, sb)] = ldw<R>(Wc, c, g, m, 2 * sa - 1, 0, 2 * sb - 1);
        }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int d = 0; d < 2; ++d) s[SO(a, b, d)] = ldw<R>(Wc, c, g, m, 2 * a - 1, 2 * b - 1, 2 * d - 1);
}

// Admissibility of a cell's FP32 traces, decided while they are stored: the density
// (c = 0) and the squared momentum (c = 1..3) of each trace point wait in the thread's
// column of a per-warp shared-memory scratch [2][NTR][32] until the energy (c = 4)
// arrives; the test is pde.c:56-66's floors, p >= 1e-12 as
// (gamma-1)(E rho - |m|^2/2) >= 1e-12 rho.
struct TraceCheck {
    float* col;  // the lane's column: [q * 32] density, [(NTR + q) * 32] |m|^2
    float g1;
    bool ok;
};

// The FP32 admissibility test of one trace point from its density, squared momentum
// |m|^2 (accumulated x, y, z in that order: m2 = mx*mx, then fma(my, my, m2), fma(mz, mz, m2))
// and energy; every operation is an explicitly rounded intrinsic, so the unfused and the fused
// stage kernels take the same decision bit for bit.
__device__ __forceinline__ bool adm_f32(float rho, float m2, float E, float g1) {
    return (rho >= 1.0e-14f) &&
           (__fmul_rn(g1, __fmaf_rn(E, rho, __fmul_rn(-0.5f, m2))) >= __fmul_rn(1.0e-12f, rho));
}

__device__ __forceinline__ void trace_check(TraceCheck* ck, int c, int q, float v) {
    float* r = ck->col + q * 32;
    float* m = ck->col + (NTR + q) * 32;
    if (c == 0) {
        *r = v;
    } else if (c == 1) {
        *m = __fmul_rn(v, v);
    } else if (c < 4) {
        *m = __fmaf_rn(v, v, *m);
    } else {
        ck->ok = ck->ok && adm_f32(*r, *m, v, ck->g1);
    }
}

// the 24 face traces of one variable into the trace array (FP32 traces: and into the
// admissibility check ck when one is given)
template <typename R>
__device__ __forceinline__ void store_traces(R* __restrict__ T, const Geo& g, long long e, int c, const R* cf,
                                             TraceCheck* ck = nullptr) {
    R tr[8];
    R* Tc = T + (long long)c * NTR * g.NE + e;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d == 0) face_traces<R, 0>(cf, tr);
        else if (d == 1) face_traces<R, 1>(cf, tr);
        else face_traces<R, 2>(cf, tr);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            Tc[(long long)(8 * d + q) * g.NE] = tr[q];
            if (sizeof(R) == sizeof(float) && ck) trace_check(ck, c, 8 * d + q, (float)tr[q]);
        }
    }
}

// density and pressure at the 24 face Gauss-point traces of one cell (what the
// Riemann solver consumes) against the floors of pde.c:56-66
__device__ __forceinline__ bool traces_admissible(const double* __restrict__ T, const Geo& g, long long e, double gm1) {
    for (int q = 0; q < NTR; ++q) {
        const double rho = T[((long long)0 * NTR + q) * g.NE + e];
        const double mx = T[((long long)1 * NTR + q) * g.NE + e];
        const double my = T[((long long)2 * NTR + q) * g.NE + e];
        const double mz = T[((long long)3 * NTR + q) * g.NE + e];
        const double E = T[((long long)4 * NTR + q) * g.NE + e];
        const double p = gm1 * (E - 0.5 * (mx * mx + my * my + mz * mz) / rho);
        if (!(rho >= 1.0e-14) || !(p >= 1.0e-12)) return false;
    }
    return true;
}

// Device-side ghost fill (what DMGlobalToLocal does for the reference's DMDA, with
// the boundary treatment of rhs_function.c's ghost loops): the stage input W (owned
// cells, SoA) copied into G with GW ghost layers on every side, each ghost the value
// its per-axis boundary map picks (periodic wrap, reflective mirror, transmissive
// copy) and a reflective ghost's wall-normal momentum negated; G is in the
// reconstruction's precision, so the FP32 form converts each value once per stage.
// One thread per ghosted cell of an x-y plane (flat index over the plane, so no block is left
// mostly idle at the end of a row), one grid row per plane.
constexpr int kGhostThreads = 256;

template <typename R>
__global__ void __launch_bounds__(kGhostThreads) k_ghost(const double* __restrict__ W, R* __restrict__ G, Geo g) {
    const int q = blockIdx.x * kGhostThreads + threadIdx.x;
    if (q >= g.gx * g.gy) return;
    const int i = q % g.gx - GW, j = q / g.gx - GW, k = blockIdx.y - GW;
    int fi = 0, fj = 0, fk = 0;
    const int mi = bmap(i, g.nx, g.bc[0], g.bc[1], &fi);
    const int mj = bmap(j, g.ny, g.bc[2], g.bc[3], &fj);
    const int mk = bmap(k, g.nz, g.bc[4], g.bc[5], &fk);
    const long long src = ((long long)mk * g.ny + mj) * g.nx + mi;
    const long long dst = ghost_index(g, i, j, k);
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        double v = __ldg(W + (long long)c * g.N + src);
        if ((c == 1 && fi) || (c == 2 && fj) || (c == 3 && fk)) v = -v;
        if constexpr (sizeof(R) == sizeof(float)) G[(long long)c * g.GN + dst] = narrow_fix(v);
        else G[(long long)c * g.GN + dst] = v;
    }
}

inline dim3 ghost_grid(const Geo& g) { return dim3(cdiv((long long)g.gx * g.gy, kGhostThreads), g.nz + 2 * GW); }

// the 33-point stencil (index map of euler_kernels.cuh) of one variable about p = &G[cell]
template <typename R>
__device__ __forceinline__ void gather33g(const R* __restrict__ p, int sy, int sz, R* s) {
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

// first-order traces (all higher coefficients zero): the fallback of
// 3d/weno4/Viscous-Multiphase-Fourth-Order/rhs_function.c:297-305
template <typename R>
__device__ __forceinline__ void store_first_order_g(const R* __restrict__ G, R* __restrict__ T, const Geo& g,
                                                    long long ge, long long e) {
#pragma unroll 1
    for (int c = 0; c < NV; ++c) {
        const R v = __ldg(G + (long long)c * g.GN + ge);
        R* Tc = T + (long long)c * NTR * g.NE + e;
        for (int q = 0; q < NTR; ++q) Tc[(long long)q * g.NE] = v;
    }
}

// FP32 reconstruction of every owned cell and of the first ghost layer (faces of the
// domain boundary), admissibility checked in dynamic shared memory
// (4 warps x 2 x NTR x 32 floats, launched only with the positivity fallback on).
__global__ void __launch_bounds__(128, 4)
    k_recon_f32(const float* __restrict__ G, float* __restrict__ T, Geo g, int recon, int pad, double gm1,
                unsigned long long* __restrict__ counters) {
    extern __shared__ float ck_dyn[];
    const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
    const int k = blockIdx.z - 1;
    if (i > g.nx || j > g.ny) return;
    const int gi = (i < 0 || i >= g.nx), gj = (j < 0 || j >= g.ny), gk = (k < 0 || k >= g.nz);
    if (gi + gj + gk > 1) return;  // edge/corner ghosts feed no face of an owned cell
    const long long e = ext_index(g, i, j, k), ge = ghost_index(g, i, j, k);
    const int sy = g.gx, sz = g.gx * g.gy;
    TraceCheck ck{ck_dyn + threadIdx.y * (2 * NTR * 32) + threadIdx.x, (float)gm1, true};
    TraceCheck* ckp = pad ? &ck : nullptr;
#pragma unroll 1
    for (int c = 0; c < NV; ++c) {
        float s[33], cf[20];
        gather33g<float>(G + (long long)c * g.GN + ge, sy, sz, s);
        if (recon == HYPE_RECON_WENO3) weno3<float>(s, cf);
        else cweno4<float>(s, recon == HYPE_RECON_LINEAR4, cf);
        store_traces<float>(T, g, e, c, cf, ckp);
    }
    if (pad && !ck.ok) {
        store_first_order_g<float>(G, T, g, ge, e);
        if (!gi && !gj && !gk) atomicAdd(&counters[1], 1ull);
    }
}

// FP64 reconstruction of the same cells, one thread per variable and cell (blockIdx.y = variable), or,
// with the positivity fallback (PAD), one per cell with the variables in turn.
// CWENO4 and R4 run on the integer pipe (cweno_fix.cuh); stencils it does not apply to, and WENO3, in FP64.
// The cells are indexed flat over the extended box: a warp of 32 x-neighbours per row left 11 % of the lanes
// idle at nx + 2 = 258 and 44 % at 18.  A variable per thread gives a small grid five times the warps (16^3:
// 183 warps of one serial 2300-instruction thread each took 87 us).  kReconThreads is small so that few blocks
// spread evenly over the SMs.  Bound: integer issue and its latencies (4000 instructions a warp, 60 % of the issue
// slots taken).  256^3, four stages: 61.1 ms at 128 registers (16 warps per SM), 63.5 at 168, 64 to 66 at 112 and
// 96; all in FP64 237.7.  62.4 since the weights are completed to one and faint polynomials looked for.
constexpr int kReconThreads = 64;

// The FP64 form of one variable in one cell: its traces and, with C, its R4 differences.  A call of its own,
// with the stencil gathered again, so that the integer form's registers do not hold it.
template <bool LINEAR>
__device__ __noinline__ void recon64_general(const double* __restrict__ p, int sy, int sz, double* __restrict__ T,
                                             double* __restrict__ C, long long NE) {
    double s[33];
    gather33g<double>(p, sy, sz, s);
    Poly64 poly;
    if constexpr (LINEAR) r4_64(s, poly);
    else cweno4_64(s, poly);
    if (T) store_traces64(poly, T, NE);
    if (C) store_grad_coeffs(poly, C, NE);
}

// What a fixed-point polynomial stays above in its cell, and what its magnitude stays below: FP32 numbers on the
// safe side, from the upper words; values outside 2^-100 to 2^117 give none
__device__ __forceinline__ float above_all(const PolyFix& p) {
    if ((unsigned)(p.top - 923) > 217u) return -INFINITY;
    return __int2float_rd((int)((p.u0 - (i64)spread_fix(p)) >> 32)) * __int_as_float((p.top - 1049 + 127) << 23);
}
__device__ __forceinline__ float below_all(const PolyFix& p) {
    if ((unsigned)(p.top - 923) > 217u) return p.top > 923 ? INFINITY : 7.9e-31f;  // 2^-100
    const u64 u = (u64)(p.u0 < 0 ? -p.u0 : p.u0);
    return __uint2float_ru((unsigned)((u + spread_fix(p)) >> 32) + 1u) * __int_as_float((p.top - 1049 + 127) << 23);
}

// The CWENO4 traces of one variable in one cell that the gate sends there; returns the bound (ends: density and
// energy, above_all; the momenta, below_all).  A call, so that k_recon64's R4 form does not hold its registers.
__device__ __noinline__ float gated_cweno4(const double* __restrict__ p, int sy, int sz, double* __restrict__ T, long long NE,
                                           bool ends) {
    double s[33];
    gather33g<double>(p, sy, sz, s);
    PolyFix fix;
    if (recon_fix<false>(s, ends, T, NE, fix)) return ends ? above_all(fix) : below_all(fix);
    recon64_general<false>(p, sy, sz, T, nullptr, NE);
    return ends ? -INFINITY : INFINITY;
}

template <int RECON, bool PAD>
__global__ void __launch_bounds__(kReconThreads, 8)
    k_recon64(const double* __restrict__ G, double* __restrict__ T, Geo g, double gm1,
              unsigned long long* __restrict__ counters, double* __restrict__ C4, const unsigned char* __restrict__ flag,
              float* __restrict__ bound) {
    const unsigned e = blockIdx.x * (unsigned)kReconThreads + threadIdx.x;
    if (e >= (unsigned)g.NE) return;
    const unsigned row = e / (unsigned)g.ex, pl = row / (unsigned)g.ey;
    const int i = (int)(e - row * (unsigned)g.ex) - 1, j = (int)(row - pl * (unsigned)g.ey) - 1, k = (int)pl - 1;
    const int gi = (i < 0 || i >= g.nx), gj = (j < 0 || j >= g.ny), gk = (k < 0 || k >= g.nz);
    if (gi + gj + gk > 1) return;  // edge/corner ghosts feed no face of an owned cell
    const long long ge = ghost_index(g, i, j, k);
    const int sy = g.gx, sz = g.gx * g.gy;
    const int c0 = PAD ? 0 : blockIdx.y, c1 = PAD ? NV : c0 + 1;
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
        double s[33];
        const double* Gc = G + (long long)c * g.GN + ge;
        double* Cc = C4 ? C4 + (long long)c * 20 * g.NE + e : nullptr;  // null without viscosity: nothing stored
        gather33g<double>(Gc, sy, sz, s);
        double* Tc = T + (long long)c * NTR * g.NE + e;
        if constexpr (RECON == HYPE_RECON_WENO3) {
            double cf[20];
            weno3<double>(s, cf);
            store_traces<double>(T, g, e, c, cf);
        } else if constexpr (RECON == HYPE_RECON_LEARNED) {
            const bool ends = c == 0 || c == 4;
            PolyFix fix;
            float b = ends ? -INFINITY : INFINITY;
            if (__ldg(flag + e)) b = gated_cweno4(Gc, sy, sz, Tc, g.NE, ends);
            else if (recon_fix<true>(s, ends, Tc, g.NE, fix)) b = ends ? above_all(fix) : below_all(fix);
            else recon64_general<true>(Gc, sy, sz, Tc, nullptr, g.NE);
            bound[c * g.NE + e] = b;
        } else {
            constexpr bool linear = RECON == HYPE_RECON_LINEAR4;
            PolyFix fix;
            if (!recon_fix<linear>(s, c == 0 || c == 4, Tc, g.NE, fix)) recon64_general<linear>(Gc, sy, sz, Tc, linear ? Cc : nullptr, g.NE);
            else if (linear && Cc) store_grad_coeffs(fix, Cc, g.NE);
        }
        // the viscous fluxes take the gradients of R4
        if (RECON != HYPE_RECON_LINEAR4 && Cc) recon64_general<true>(Gc, sy, sz, nullptr, Cc, g.NE);
    }
    if (PAD && !traces_admissible(T, g, e, gm1)) {
        store_first_order_g<double>(G, T, g, ge, e);
        if (!gi && !gj && !gk) atomicAdd(&counters[1], 1ull);
    }
}

static void launch_recon64(const Geo& g, const double* G, double* T, int recon, int pad, double gm1,
                           unsigned long long* counters, double* C4, cudaStream_t st) {
    const dim3 gr(cdiv(g.NE, kReconThreads), pad ? 1 : NV);
    auto go = [&](auto kern) { kern<<<gr, kReconThreads, 0, st>>>(G, T, g, gm1, counters, C4, nullptr, nullptr); };
    if (recon == HYPE_RECON_WENO3) pad ? go(k_recon64<HYPE_RECON_WENO3, true>) : go(k_recon64<HYPE_RECON_WENO3, false>);
    else if (recon == HYPE_RECON_LINEAR4) pad ? go(k_recon64<HYPE_RECON_LINEAR4, true>) : go(k_recon64<HYPE_RECON_LINEAR4, false>);
    else pad ? go(k_recon64<HYPE_RECON_CWENO4, true>) : go(k_recon64<HYPE_RECON_CWENO4, false>);
}

// The gated FP64 reconstruction's second pass.  k_recon64 took each variable through CWENO4 or R4 by the cell's flag
// and left a bound of its polynomial; where the bounds keep density and pressure above the floors (all but a few
// cells), the 24 traces need not be read.  A cell whose R4 traces break them is redone here with CWENO4, then first
// order with the fallback.
// 256^3 blast: one kernel for scoring, a cell's variables in turn, and a check that read its 120 traces back, ran at
// 104.8 M cell-updates/s, below CWENO4 without a gate; a block of 32 cells x 5 variables for all of it at 134.7 M; this,
// with k_gate's flags, 197.8 M.
constexpr int kGatedThreads = 128;
__global__ void __launch_bounds__(kGatedThreads)
    k_gated_check(const double* __restrict__ G, double* __restrict__ T, Geo g, double gm1, int pad,
                  const unsigned char* __restrict__ flag, const float* __restrict__ bound,
                  unsigned long long* __restrict__ counters) {
    const unsigned e = blockIdx.x * (unsigned)kGatedThreads + threadIdx.x, row = e / (unsigned)g.ex, pl = row / (unsigned)g.ey;
    const int i = (int)(e - row * (unsigned)g.ex) - 1, j = (int)(row - pl * (unsigned)g.ey) - 1, k = (int)pl - 1;
    const int gi = (i < 0 || i >= g.nx), gj = (j < 0 || j >= g.ny), gk = (k < 0 || k >= g.nz);
    const bool active = e < (unsigned)g.NE && gi + gj + gk <= 1, owned = active && !(gi | gj | gk);
    const bool full = active && __ldg(flag + e);
    if (active) {
        const float* b = bound + e;
        const float rho = __ldg(b), mx = __ldg(b + g.NE), my = __ldg(b + 2 * g.NE), mz = __ldg(b + 3 * g.NE), E = __ldg(b + 4 * g.NE);
        const float kin = 0.5f * (mx * mx + my * my + mz * mz) / rho;
        // on the safe side of the FP32 roundings; false for infinities and NaN
        const bool clear = rho > 1.001e-14f && (E - kin) - 1e-4f * (E + kin) > 1.001e-12f / (float)gm1;
        bool ok = clear || traces_admissible(T, g, e, gm1);
        const long long ge = ghost_index(g, i, j, k);
        if (!ok && !full) {
#pragma unroll 1
            for (int c = 0; c < NV; ++c)
                gated_cweno4(G + (long long)c * g.GN + ge, g.gx, g.gx * g.gy, T + (long long)c * NTR * g.NE + e, g.NE, c == 0 || c == 4);
            ok = traces_admissible(T, g, e, gm1);
        }
        if (!ok && pad) {  // CWENO4 itself inadmissible
            store_first_order_g<double>(G, T, g, ge, e);
            if (owned) atomicAdd(&counters[1], 1ull);
        }
    }
    const int flagged = __syncthreads_count(full && owned);
    if (threadIdx.x == 0 && flagged) atomicAdd(&counters[0], (unsigned long long)flagged);
}

// Indicator-gated reconstruction: the network scores the cell from its three
// directional 5-point stencils; flagged or low-confidence cells take the full
// CWENO4, the others the linear R4 -- unless the linear traces give a density
// or pressure below the floors at any face Gauss point, in which case the cell
// is redone with CWENO4 (positivity fallback).
__global__ void __launch_bounds__(128, 4)
    k_recon_learned(const float* __restrict__ G, float* __restrict__ T, Geo g, const mlp::MmaWeights* __restrict__ wts,
                    float logit_thr, double gm1, int pad, unsigned long long* __restrict__ counters) {
    // per warp: the staged network inputs, later the admissibility scratch
    static_assert(mlp::ROWS * mlp::RSTRIDE * sizeof(__nv_bfloat16) >= 2 * NTR * 32 * sizeof(float), "scratch");
    __shared__ __align__(16) __nv_bfloat16 rows[4][mlp::ROWS * mlp::RSTRIDE];
    __shared__ float lg[4][mlp::ROWS];
    __shared__ unsigned cnt[2];
    if (threadIdx.x == 0 && threadIdx.y == 0) cnt[0] = cnt[1] = 0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
    const int k = blockIdx.z - 1;
    bool active = !(i > g.nx || j > g.ny);
    const int gi = (i < 0 || i >= g.nx), gj = (j < 0 || j >= g.ny), gk = (k < 0 || k >= g.nz);
    active = active && (gi + gj + gk <= 1);
    const long long ge = active ? ghost_index(g, i, j, k) : 0;
    const int sy = g.gx, sz = g.gx * g.gy;
    // features of the warp's 32 cells (3 rows each) staged as BF16, scored on the tensor cores
    __nv_bfloat16* my_rows = rows[threadIdx.y] + threadIdx.x * 3 * mlp::RSTRIDE;
    float sc[NV];
    if (active) {
        const float rho = __ldg(G + ge), E = __ldg(G + 4 * g.GN + ge);
#pragma unroll
        for (int c = 0; c < NV; ++c) sc[c] = mlp::var_scale<float>(c, rho, E);
    }
#pragma unroll 1
    for (int d = 0; d < 3; ++d) {
        float x[mlp::NIN];
        const int st = d == 0 ? 1 : d == 1 ? sy : sz;
        if (active) {
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const float* p = G + (long long)c * g.GN + ge;
                const float s5[5] = {__ldg(p - 2 * st), __ldg(p - st), __ldg(p), __ldg(p + st), __ldg(p + 2 * st)};
                mlp::normalise5(s5, sc[c], x + c * 5);
            }
        }
        mlp::stage_row(my_rows + d * mlp::RSTRIDE, x, active);
    }
    __syncthreads();  // counters cleared, rows staged
    mlp::warp_logits(wts, rows[threadIdx.y], lg[threadIdx.y]);
    __syncwarp();
    const float best = fmaxf(lg[threadIdx.y][threadIdx.x * 3], fmaxf(lg[threadIdx.y][threadIdx.x * 3 + 1],
                                                                       lg[threadIdx.y][threadIdx.x * 3 + 2]));
    if (active) {
        const long long e = ext_index(g, i, j, k);
        TraceCheck ck{reinterpret_cast<float*>(rows[threadIdx.y]) + threadIdx.x, (float)gm1, true};
        bool full = best > logit_thr;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            ck.ok = true;
#pragma unroll 1
            for (int c = 0; c < NV; ++c) {
                float s[33], cf[20];
                gather33g<float>(G + (long long)c * g.GN + ge, sy, sz, s);
                cweno4<float>(s, !full, cf);
                store_traces<float>(T, g, e, c, cf, &ck);
            }
            if (ck.ok) break;
            if (full) {  // CWENO4 itself inadmissible: first order (when enabled)
                if (pad) {
                    store_first_order_g<float>(G, T, g, ge, e);
                    if (!gi && !gj && !gk) atomicAdd(&cnt[1], 1u);
                }
                break;
            }
            full = true;  // the R4 traces broke positivity: redo the cell with CWENO4
        }
        if (full && !gi && !gj && !gk && best > logit_thr) atomicAdd(&cnt[0], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        if (cnt[0]) atomicAdd(&counters[0], (unsigned long long)cnt[0]);
        if (cnt[1]) atomicAdd(&counters[1], (unsigned long long)cnt[1]);
    }
}

// Indicator training data: for every stride-th owned cell, the three directional
// normalised stencils (X[s][3][25]) and D[s], the largest change that the nonlinear
// CWENO4 weights make to a face trace relative to the linear R4 polynomial, over the
// 5 variables and 24 traces, in units of the variable's magnitude in the cell (labels:
// D > tau).
__global__ void __launch_bounds__(128) k_features(const double* __restrict__ W, Geo g, long long stride, long long ns,
                                                  float* __restrict__ X, float* __restrict__ D) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s >= ns) return;
    const long long cell = s * stride;
    const int i = (int)(cell % g.nx), j = (int)((cell / g.nx) % g.ny), k = (int)(cell / ((long long)g.nx * g.ny));
    StencilMap m;
    make_map(g, i, j, k, m);
    const double rho = ldw<double, double>(W, 0, g, m, 0, 0, 0), E = ldw<double, double>(W + 4 * g.N, 4, g, m, 0, 0, 0);
    double dmax = 0.0;
#pragma unroll 1
    for (int c = 0; c < NV; ++c) {
        double st[33], cf[20], cl[20], ta[8], tb[8];
        gather33<double, double>(W + (long long)c * g.N, c, g, m, st);
        Poly64 poly;
        cweno4_64(st, poly);
        coeffs64(poly, cf);
        r4_64(st, poly);
        coeffs64(poly, cl);
        const double scale = mlp::var_scale<double>(c, rho, E) + 1e-30;
        double dd = 0.0;
        face_traces<double, 0>(cf, ta);
        face_traces<double, 0>(cl, tb);
        for (int q = 0; q < 8; ++q) dd = fmax(dd, fabs(ta[q] - tb[q]));
        face_traces<double, 1>(cf, ta);
        face_traces<double, 1>(cl, tb);
        for (int q = 0; q < 8; ++q) dd = fmax(dd, fabs(ta[q] - tb[q]));
        face_traces<double, 2>(cf, ta);
        face_traces<double, 2>(cl, tb);
        for (int q = 0; q < 8; ++q) dd = fmax(dd, fabs(ta[q] - tb[q]));
        dmax = fmax(dmax, dd / scale);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float s5[5] = {(float)st[S1(d, -2)], (float)st[S1(d, -1)], (float)st[0], (float)st[S1(d, 1)],
                                 (float)st[S1(d, 2)]};
            mlp::normalise5(s5, (float)mlp::var_scale<double>(c, rho, E), X + (s * 3 + d) * mlp::NIN + c * 5);
        }
    }
    D[s] = (float)dmax;
}

__device__ __forceinline__ void atomic_max_pos(unsigned long long* a, double v) {
    atomicMax(a, (unsigned long long)__double_as_longlong(v));
}

// the FP32 face fluxes of direction D, one thread per face; face (i, j, k) is the low side of cell (i, j, k) and
// runs to n along D
template <int D, int FLUX>
__global__ void __launch_bounds__(128) k_faces_f32(const float* __restrict__ T, double* __restrict__ F, Geo g, double gamma,
                                                   DevScalars* __restrict__ ds, int slot) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    const int fx = g.nx + (D == 0), fy = g.ny + (D == 1);
    double smax = 0.0;
    bool bad = false;
    const bool active = (i < fx && j < fy);
    if (active) {
        const long long eR = ext_index(g, i, j, k);
        const long long eL = ext_index(g, i - (D == 0), j - (D == 1), k - (D == 2));
        float acc[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) acc[c] = 0.0f;
        const float gm = (float)gamma, gm1 = (float)(gamma - 1.0);
#pragma unroll
        for (int gp = 0; gp < 4; ++gp) {
            float QL[NV], QR[NV], fl[NV];
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                QL[c] = T[((long long)c * NTR + (2 * D + 1) * 4 + gp) * g.NE + eL];
                QR[c] = T[((long long)c * NTR + (2 * D) * 4 + gp) * g.NE + eR];
            }
            // Rusanov's 1/2 goes into the Gauss weight 1/4
            float s;
            if constexpr (FLUX == HYPE_FLUX_RUSANOV) s = rusanov<float, D>(QL, QR, gm, gm1, fl, bad);
            else s = face_solver<float, D, FLUX>(QL, QR, gm, gm1, fl, bad);
            smax = fmax(smax, (double)s);
            const float wq = FLUX == HYPE_FLUX_RUSANOV ? 0.125f : 0.25f;
#pragma unroll
            for (int c = 0; c < NV; ++c) acc[c] += wq * fl[c];
        }
        const long long nf = (long long)fx * fy * (g.nz + (D == 2));
        const long long f = ((long long)k * fy + j) * fx + i;
#pragma unroll
        for (int c = 0; c < NV; ++c) F[c * nf + f] = (double)acc[c];
        if (bad) {
            const int ci = i < g.nx ? i : g.nx - 1, cj = j < g.ny ? j : g.ny - 1, ck = k < g.nz ? k : g.nz - 1;
            atomicMin(&ds->bad, (unsigned long long)(((long long)ck * g.ny + cj) * g.nx + ci));
        }
    }
    // warp max, one atomic per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) smax = fmax(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    if ((threadIdx.x & 31) == 0 && smax > 0.0) atomic_max_pos(&ds->smax_bits[slot], smax);
}

// The faces normal to D, indexed flat: face (i, j, k) is the low side of cell (i, j, k) and runs to n
// along D.  Its number, its two cells in the trace array and the cell an inadmissible state is reported at.
template <int D>
struct FaceAt {
    unsigned nf, f;
    int i, j, k;
    __device__ __forceinline__ FaceAt(const Geo& g, unsigned face) : f(face) {
        const unsigned fx = g.nx + (D == 0), fy = g.ny + (D == 1), fz = g.nz + (D == 2);
        nf = fx * fy * fz;
        const unsigned row = f / fx, pl = row / fy;
        i = (int)(f - row * fx);
        j = (int)(row - pl * fy);
        k = (int)pl;
    }
    __device__ __forceinline__ long long hi(const Geo& g) const { return ext_index(g, i, j, k); }
    __device__ __forceinline__ long long lo(const Geo& g) const {
        return ext_index(g, i - (D == 0), j - (D == 1), k - (D == 2));
    }
    __device__ __forceinline__ void report(const Geo& g, DevScalars* ds) const {
        const int ci = i < g.nx ? i : g.nx - 1, cj = j < g.ny ? j : g.ny - 1, ck = k < g.nz ? k : g.nz - 1;
        atomicMin(&ds->bad, (unsigned long long)(((long long)ck * g.ny + cj) * g.nx + ci));
    }
};

// the warp's maximum of a non-negative number, decided on the bit pattern; a lane with a NaN does not count
__device__ __forceinline__ double warp_max_pos(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max_num(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// The maximum only grows while a kernel runs: a warp whose value does not exceed what it reads leaves it
// alone (one atomic per warp to one address would serialise millions of them).
__device__ __forceinline__ void raise_max(unsigned long long* slot, double v) {
    if (v > 0.0 && (unsigned long long)__double_as_longlong(v) > *(volatile unsigned long long*)slot) atomic_max_pos(slot, v);
}

// FP64 face fluxes, all three directions in one launch (blockIdx.y = direction).  A block is 32 faces x
// the 4 Gauss points of the 2x2 rule, one point per warp: a quarter of the registers of a thread per face,
// four times the warps on a small grid (16^3: three launches of one 16 us wave each), the traces of a warp
// contiguous in x and the four fluxes summed through shared memory.
// Bound: FP64 issue still, 26 operations per Rusanov solve with the side states and the sum over the points on the
// integer pipe (about 1100 integer instructions beside them): 256^3, four stages 97.1 -> 38.6 ms.
template <int D, int FLUX>
__device__ __forceinline__ void faces64(const double* __restrict__ T, double* __restrict__ F, const Geo& g, double gamma,
                                        DevScalars* __restrict__ ds, int slot, double (*sh)[NV][32]) {
    const int lane = threadIdx.x & 31, gp = threadIdx.x >> 5;
    const FaceAt<D> at(g, blockIdx.x * 32u + lane);
    if (blockIdx.x * 32u >= at.nf) return;  // the grid is as wide as the direction with the most faces
    double smax = 0.0;
    if (at.f < at.nf) {
        const double* TL = T + ((2 * D + 1) * 4 + gp) * g.NE + at.lo(g);
        const double* TR = T + (2 * D * 4 + gp) * g.NE + at.hi(g);
        double QL[NV], QR[NV], fl[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            QL[c] = __ldg(TL + c * NTR * g.NE);
            QR[c] = __ldg(TR + c * NTR * g.NE);
        }
        bool bad = false;
        if constexpr (FLUX == HYPE_FLUX_RUSANOV) smax = rusanov_fix<D>(QL, QR, gamma, gamma - 1.0, fl, bad);
        else smax = face_solver<double, D, FLUX>(QL, QR, gamma, gamma - 1.0, fl, bad);
#pragma unroll
        for (int c = 0; c < NV; ++c) sh[gp][c][lane] = fl[c];
        if (bad) at.report(g, ds);
    }
    smax = warp_max_pos(smax);
    if (lane == 0) raise_max(&ds->smax_bits[slot], smax);
    __syncthreads();
    // Rusanov's 1/2 goes into the Gauss weight 1/4
    constexpr int shift = FLUX == HYPE_FLUX_RUSANOV ? 3 : 2;
    for (int c = gp; c < NV; c += 4)
        if (at.f < at.nf) F[(long long)c * at.nf + at.f] = sum4(sh[0][c][lane], sh[1][c][lane], sh[2][c][lane], sh[3][c][lane], shift);
}

template <int FLUX>
__global__ void __launch_bounds__(128) k_faces64(const double* __restrict__ T, double* __restrict__ Fx,
                                                 double* __restrict__ Fy, double* __restrict__ Fz, Geo g, double gamma,
                                                 DevScalars* __restrict__ ds, int slot) {
    __shared__ double sh[4][NV][32];
    if (blockIdx.y == 0) faces64<0, FLUX>(T, Fx, g, gamma, ds, slot, sh);
    else if (blockIdx.y == 1) faces64<1, FLUX>(T, Fy, g, gamma, ds, slot, sh);
    else faces64<2, FLUX>(T, Fz, g, gamma, ds, slot, sh);
}

// Navier-Stokes faces: the inviscid flux plus, at each Gauss point, half of both sides' viscous fluxes
// (PDEViscRiemannSolver, Navier-Stokes-3D/pde.c:386-404; rhs_function.c:310-316), laid out as faces64: a Gauss
// point per warp.  Bound: FP64 issue (120 operations a warp) and the integer pipe's 5000 instructions beside it.
// 96^3, an RHS: 3.71 ms as a thread per face all in FP64 (203 operations a point), 4.01 with the gradients as
// integers (180 registers, 8 warps per SM, which fill neither pipe), 3.59 a point per warp at 80 registers, 2.58
// with the 22 gradient forms of a face shared out among the four warps.
struct ViscShared {
    double flux[4][NV][32];
    i64 form[2 * NFORM][4][32];
    int top[2][NV][32];
};
template <int D, int FLUX>
__device__ __forceinline__ void faces_visc64(const double* __restrict__ T, double* __restrict__ F, const Geo& g,
                                             double gamma, DevScalars* __restrict__ ds, int slot,
                                             const double* __restrict__ C4, const Visc& vp, ViscShared& sh) {
    constexpr int T1 = D == 0 ? 1 : 0, T2 = D == 2 ? 1 : 2;
    const int lane = threadIdx.x & 31, gp = threadIdx.x >> 5;
    const FaceAt<D> at(g, blockIdx.x * 32u + lane);
    if (blockIdx.x * 32u >= at.nf) return;  // the grid is as wide as the direction with the most faces
    double smax = 0.0, smaxv = 0.0;
    const bool in = at.f < at.nf;
    const long long eR = in ? at.hi(g) : 0, eL = in ? at.lo(g) : 0;
    if (in) {
        auto form = [&](auto k) {
            constexpr int K = decltype(k)::value, side = K / NFORM;
            i64 P, Q, R, S;
            side_form64<D, side ? -1 : 1, K % NFORM>(C4 + (side ? eR : eL), g.NE, P, Q, R, S);
            sh.form[K][0][lane] = P;
            sh.form[K][1][lane] = Q;
            sh.form[K][2][lane] = R;
            sh.form[K][3][lane] = S;
        };
        auto forms = [&](auto... k) { (form(k), ...); };
#define FORM(k) std::integral_constant<int, k>{}
        if (gp == 0) forms(FORM(0), FORM(4), FORM(8), FORM(12), FORM(16), FORM(20));
        else if (gp == 1) forms(FORM(1), FORM(5), FORM(9), FORM(13), FORM(17), FORM(21));
        else if (gp == 2) forms(FORM(2), FORM(6), FORM(10), FORM(14), FORM(18));
        else forms(FORM(3), FORM(7), FORM(11), FORM(15), FORM(19));
#undef FORM
        for (int q = gp; q < 2 * NV; q += 4)
            sh.top[q / NV][q % NV][lane] =
                (int)__double_as_longlong(__ldg(C4 + ((q % NV) * 20 + 19) * g.NE + (q < NV ? eL : eR)));
    }
    __syncthreads();
    if (in) {
        const double* TL = T + ((2 * D + 1) * 4 + gp) * g.NE + eL;
        const double* TR = T + (2 * D * 4 + gp) * g.NE + eR;
        double QL[NV], QR[NV], fl[NV], av[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            QL[c] = __ldg(TL + c * NTR * g.NE);
            QR[c] = __ldg(TR + c * NTR * g.NE);
        }
        bool bad = false;
        if constexpr (FLUX == HYPE_FLUX_RUSANOV) smax = rusanov_fix<D>(QL, QR, gamma, gamma - 1.0, fl, bad);
        else smax = face_solver<double, D, FLUX>(QL, QR, gamma, gamma - 1.0, fl, bad);
        const double kmu = vp.kc / vp.mu;
        const i64 n1 = (gp & 2) ? 0 : -1, n2 = (gp & 1) ? 0 : -1;  // all ones where the point's coordinate is negative
        auto grads = [&](int side) {
            return [&, side](int k) {
                const i64(*f)[32] = sh.form[side * NFORM + k];
                const i64 RS = f[2][lane] + ((f[3][lane] ^ n1) - n1);
                const int var = k < 3 ? 0 : k < 6 ? 1 + D : k < 8 ? 1 + T1 : k < 10 ? 1 + T2 : 4;
                return double_of(f[0][lane] + ((f[1][lane] ^ n1) - n1) + ((RS ^ n2) - n2), sh.top[side][var][lane]);
            };
        };
        smaxv = visc_point64<D>(QL, grads(0), gamma - 1.0, kmu, av);
        smaxv = vp.vmax * max_num(smaxv, visc_point64<D>(QR, grads(1), gamma - 1.0, kmu, av));
        // weight 1/4, both sides' mean, twice the gradients times h: mu / (16 h), in units of the inviscid weight
        constexpr double wq = FLUX == HYPE_FLUX_RUSANOV ? 0.125 : 0.25;
        const double wv = -(1. / 16.) / wq * vp.mu * vp.r1_h;
        fl[1 + D] = fma(wv, av[0], fl[1 + D]);
        fl[1 + T1] = fma(wv, av[1], fl[1 + T1]);
        fl[1 + T2] = fma(wv, av[2], fl[1 + T2]);
        fl[4] = fma(wv, av[3], fl[4]);
#pragma unroll
        for (int c = 0; c < NV; ++c) sh.flux[gp][c][lane] = fl[c];
        if (bad) at.report(g, ds);
    }
    smax = warp_max_pos(smax);
    smaxv = warp_max_pos(smaxv);
    if (lane == 0) {
        raise_max(&ds->smax_bits[slot], smax);
        raise_max(&ds->smaxv_bits[slot], smaxv);
    }
    __syncthreads();
    constexpr int shift = FLUX == HYPE_FLUX_RUSANOV ? 3 : 2;
    for (int c = gp; c < NV; c += 4)
        if (at.f < at.nf) F[(long long)c * at.nf + at.f] = sum4(sh.flux[0][c][lane], sh.flux[1][c][lane], sh.flux[2][c][lane],
                                                                   sh.flux[3][c][lane], shift);
}

template <int FLUX>
__global__ void __launch_bounds__(128, 5) k_faces_visc64(const double* __restrict__ T, double* __restrict__ Fx,
                                                      double* __restrict__ Fy, double* __restrict__ Fz, Geo g, double gamma,
                                                      DevScalars* __restrict__ ds, int slot, const double* __restrict__ C4,
                                                      Visc vp) {
    __shared__ ViscShared sh;
    if (blockIdx.y == 0) faces_visc64<0, FLUX>(T, Fx, g, gamma, ds, slot, C4, vp, sh);
    else if (blockIdx.y == 1) faces_visc64<1, FLUX>(T, Fy, g, gamma, ds, slot, C4, vp, sh);
    else faces_visc64<2, FLUX>(T, Fz, g, gamma, ds, slot, C4, vp, sh);
}

// stage combination: out = a*U + b*W + (c*dt)*L   (L = divergence of the face fluxes)
struct Stage {
    double a, b, c;
    int rhs_only;
};

// the FP32 form's divergence -(1/h)(dx + dy + dz), dx = F(i+1/2) - F(i-1/2) etc., as explicitly rounded operations
// in a fixed order, the x and y part first (the fused stage kernel forms the two parts one plane apart): its
// face fluxes are FP32 values, differenced and scaled in FP32
// (neighbouring fluxes lie within a factor 2 of each other in smooth flow, where the FP32
// differences are exact); only the stage combination is FP64
__device__ __forceinline__ float div_xy_f(float dx, float dy, float r1_h) {
    return __fmaf_rn(-r1_h, dy, __fmul_rn(-r1_h, dx));
}
__device__ __forceinline__ float div_z_f(float pxy, float dz, float r1_h) { return __fmaf_rn(-r1_h, dz, pxy); }

// the SSP stage value a U + b W + (c dt) L (b = 1 when a = 0), explicitly rounded
__device__ __forceinline__ double stage_value(const Stage& st, double cdt, double u, double w, double L) {
    if (st.rhs_only) return L;
    if (st.a == 0.0) return __fma_rn(cdt, L, w);
    return __fma_rn(cdt, L, __fma_rn(st.b, w, __dmul_rn(st.a, u)));
}

// U, W and out may be one array (in-place stages), so they carry no __restrict__; a thread per cell and
// variable (blockIdx.y) keeps the loads of one from waiting for the stores of another (16^3: 9.5 us with a
// cell per thread).  F32: the face fluxes hold FP32 values (the FP32 form); the divergence is formed in FP32.
// FP64: bound by FP64 issue, so the six fluxes are summed as integers and the factor c dt / h is formed once a
// block: 2 to 4 FP64 operations for 9 to 11.  256^3, four stages: 7.5 -> 3.4 ms.
constexpr int kUpdateThreads = 256;

template <bool F32 = false>
__global__ void __launch_bounds__(kUpdateThreads) k_update(const double* __restrict__ Fx, const double* __restrict__ Fy,
                                                           const double* __restrict__ Fz, const double* U,
                                                           const double* W, double* out, Geo g, double r1_h,
                                                           Stage st, const DevScalars* __restrict__ ds) {
    __shared__ double factor;  // c dt, or -c dt / h of the FP64 form
    const unsigned cell = blockIdx.x * (unsigned)kUpdateThreads + threadIdx.x;
    const bool inside = cell < (unsigned)g.N;
    const unsigned row = cell / (unsigned)g.nx, k = row / (unsigned)g.ny;
    const long long c = blockIdx.y;
    const long long nfx = (long long)(g.nx + 1) * g.ny * g.nz, nfy = (long long)g.nx * (g.ny + 1) * g.nz,
                    nfz = (long long)g.nx * g.ny * (g.nz + 1);
    Fx += c * nfx + cell + row;                    // (k ny + j) (nx + 1) + i
    Fy += c * nfy + cell + k * (unsigned)g.nx;     // (k (ny + 1) + j) nx + i
    Fz += c * nfz + cell;
    const bool with_u = !st.rhs_only && __double2hiint(st.a) != 0;
    double f[6] = {}, u = 0.0, w = 0.0;
    if (inside) {  // everything is under way before the block waits for its factor
        f[0] = Fx[1]; f[1] = Fx[0]; f[2] = Fy[g.nx]; f[3] = Fy[0]; f[4] = Fz[(long long)g.nx * g.ny]; f[5] = Fz[0];
        if (with_u) u = U[c * g.N + cell];
        if (!st.rhs_only) w = W[c * g.N + cell];
    }
    if (threadIdx.x == 0) {
        const double cdt = st.rhs_only ? 1.0 : st.c * ds->dt;
        factor = F32 ? cdt : -cdt * r1_h;
    }
    __syncthreads();
    if (!inside) return;
    if constexpr (F32) {
        // exact: the fluxes are FP32 values.  By instruction the six conversions and the stage's comparison were
        // eight FP64 issues of eleven (HLLC 128^3, a launch 228 us; a cell per thread, comparison shared 150)
        float q[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) q[i] = narrow_fix(f[i]);
        const float r1hf = (float)r1_h;
        const double L = df_f2d(div_z_f(div_xy_f(q[0] - q[1], q[2] - q[3], r1hf), q[4] - q[5], r1hf));
        out[c * g.N + cell] = st.rhs_only ? L : __fma_rn(factor, L, with_u ? __fma_rn(st.b, w, __dmul_rn(st.a, u)) : w);
    } else {
        const double L = sum_differences(f[0], f[1], f[2], f[3], f[4], f[5]);
        if (with_u) w = fma(st.b, w, st.a * u);
        out[c * g.N + cell] = fma(factor, L, w);  // RHS-only: w = 0
    }
}
inline dim3 update_grid(const Geo& g) { return dim3(cdiv(g.N, kUpdateThreads), NV); }

// ---------------------------------------------------------------- fused FP32 stage
// One pass per RK stage for the FP32 reconstruction + Rusanov flux form: reconstruction of
// every variable, the 24 face traces, the Rusanov solves at the face Gauss points, the flux
// divergence, the wave-speed maximum, the admissibility word and the SSP stage combination,
// with the face traces kept in shared memory (the unfused kernels write 120 traces per cell to
// HBM and read them back: 960 B per cell-stage of FP32 traffic).  It follows the loop
// structure of 3d/weno4/Navier-Stokes-3D/rhs_function.c:183-433 (reconstruct, evaluate the
// face traces, solve per face Gauss point, difference) over tiles instead of the whole box.
//
// Layout: a block is FS_TW warps of 32 lanes.  Lane l of warp w holds cell
// (i0 + l - 1, j0 + w - 1) of an x-y tile: lanes 1..30 and warps 1..FS_TW-2 are the owned
// cells, lane 0 / 31 and warp 0 / FS_TW-1 the one-cell ring whose traces the tile's boundary
// faces need (the ring is reconstructed again by the neighbouring tile: 80 ring cells beside
// the 300 owned ones per plane).  The block marches its tile along z; the +z traces of a plane stay in the
// thread's registers as the -z side of the next plane's z faces, and each cell's divergence
// is completed one plane later, when its +z face flux exists.  Blocks are persistent, one per
// SM (the trace and flux arrays take 188 KB of shared memory), and split the tiles' planes into equal
// contiguous runs: a run re-reconstructs one plane below and one above it.
// Every arithmetic step is the unfused kernels' (cweno4 / weno3, face_traces, rusanov, the
// admissibility test and the divergence use the same device functions and explicit roundings),
// so both paths give bit-identical results.
constexpr int FS_TW = 12;                        // warps per block (at most 168 registers per thread)
constexpr int FS_NT = 32 * FS_TW;                // 384 threads
constexpr int FS_OX = 30, FS_OY = FS_TW - 2;     // owned tile: 30 x 10 cells
constexpr int FS_NQ = NV * NTR;                  // traces per cell
// traces [c][q][thread] and the -y face fluxes [c][thread] (FP32): 192,000 B, which leaves 60 KB of
// the SM's L1 for the stencil gathers
constexpr size_t FS_SMEM = sizeof(float) * (FS_NQ + NV) * FS_NT;

__host__ __device__ inline long long fs_tiles_x(int nx) { return (nx + FS_OX - 1) / FS_OX; }
__host__ __device__ inline long long fs_tiles_y(int ny) { return (ny + FS_OY - 1) / FS_OY; }

// one Rusanov face (weight 1/8 per Gauss point, as k_faces): L side trace q0L.., R side q0R..
// read from the shared trace array (columns tL, tR) or, for the z faces' low side, from registers
__device__ __forceinline__ void fs_face(const float* __restrict__ S, int tL, int tR, int qL, int qR,
                                        const float (*zl)[4], float gm, float gm1, float* Fd, float& smax,
                                        bool& bad, int D) {
    float acc[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) acc[c] = 0.0f;
#pragma unroll
    for (int gp = 0; gp < 4; ++gp) {
        float QL[NV], QR[NV], fl[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            QL[c] = zl ? zl[c][gp] : S[(c * NTR + qL + gp) * FS_NT + tL];
            QR[c] = S[(c * NTR + qR + gp) * FS_NT + tR];
        }
        float s;
        if (D == 0) s = rusanov<float, 0>(QL, QR, gm, gm1, fl, bad);
        else if (D == 1) s = rusanov<float, 1>(QL, QR, gm, gm1, fl, bad);
        else s = rusanov<float, 2>(QL, QR, gm, gm1, fl, bad);
        smax = fmaxf(smax, s);
#pragma unroll
        for (int c = 0; c < NV; ++c) acc[c] += 0.125f * fl[c];
    }
#pragma unroll
    for (int c = 0; c < NV; ++c) Fd[c] = acc[c];
}

// a hint that the line holding *a will be read soon (into L2); a must lie inside its array
__device__ __forceinline__ void prefetch_l2(const void* a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }

__device__ __forceinline__ void fs_bad(DevScalars* ds, const Geo& g, int i, int j, int k) {
    const int ci = i < g.nx ? i : g.nx - 1, cj = j < g.ny ? j : g.ny - 1, ck = k < g.nz ? k : g.nz - 1;
    atomicMin(&ds->bad, (unsigned long long)(((long long)ck * g.ny + cj) * g.nx + ci));
}

// one cell's 24 traces of every variable into its column of the shared array (linear: R4)
__device__ __forceinline__ void fs_recon_cell(float* __restrict__ S, const float* __restrict__ G, const Geo& g,
                                              long long ge, int t, bool linear, bool weno) {
    const int sy = g.gx, sz = g.gx * g.gy;
    // unrolled, so that one variable's gathers are under way while another is computed: with 12 warps per SM the
    // kernel waits for them (256^3 blast, a stage 5.56 ms rolled, 5.18 unrolled, 5.10 with the planes ahead
    // prefetched)
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        float s[33], cf[20], tr[8];
        gather33g<float>(G + (long long)c * g.GN + ge, sy, sz, s);
        if (weno) weno3<float>(s, cf);
        else cweno4<float>(s, linear, cf);
        float* Sc = S + (c * NTR) * FS_NT + t;
        face_traces<float, 0>(cf, tr);
#pragma unroll
        for (int q = 0; q < 8; ++q) Sc[q * FS_NT] = tr[q];
        face_traces<float, 1>(cf, tr);
#pragma unroll
        for (int q = 0; q < 8; ++q) Sc[(8 + q) * FS_NT] = tr[q];
        face_traces<float, 2>(cf, tr);
#pragma unroll
        for (int q = 0; q < 8; ++q) Sc[(16 + q) * FS_NT] = tr[q];
    }
}

// the cell's 24 traces (its own column) against the density / pressure floors
__device__ __forceinline__ bool fs_admissible(const float* __restrict__ S, int t, float gm1) {
    bool ok = true;
#pragma unroll 4
    for (int q = 0; q < NTR; ++q) {
        const float rho = S[(0 * NTR + q) * FS_NT + t];
        float m2 = __fmul_rn(S[(1 * NTR + q) * FS_NT + t], S[(1 * NTR + q) * FS_NT + t]);
        m2 = __fmaf_rn(S[(2 * NTR + q) * FS_NT + t], S[(2 * NTR + q) * FS_NT + t], m2);
        m2 = __fmaf_rn(S[(3 * NTR + q) * FS_NT + t], S[(3 * NTR + q) * FS_NT + t], m2);
        ok = ok && adm_f32(rho, m2, S[(4 * NTR + q) * FS_NT + t], gm1);
    }
    return ok;
}

// The learned gate of the fused FP32 stage and of the FP64 reconstruction, scored ahead of them from the ghosted copy: one
// byte per extended cell, 1 where the network's largest directional logit exceeds the threshold.
// Scored are the cells the stage reconstructs (the owned cells and the one-cell frame without its
// edges and corners, which keep the zero the array is created with).  The features, their BF16
// rounding and the tensor-core scoring are k_recon_learned's, so the flags are that kernel's
// decisions bit for bit.  Block: 32 x 4 cells of one x-y plane, as k_recon_learned.
template <typename R>
__global__ void __launch_bounds__(128) k_gate(const R* __restrict__ G, unsigned char* __restrict__ flag, Geo g,
                                              const mlp::MmaWeights* __restrict__ wts, float logit_thr) {
    auto ld = [](const R* p) {
        if constexpr (sizeof(R) == sizeof(double)) return narrow_fix(__ldg(p));
        else return __ldg(p);
    };
    __shared__ __align__(16) __nv_bfloat16 rows[4][mlp::ROWS * mlp::RSTRIDE];
    __shared__ float lg[4][mlp::ROWS];
    const int i = blockIdx.x * blockDim.x + threadIdx.x - 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y - 1;
    const int k = blockIdx.z - 1;
    const int gi = (i < 0 || i >= g.nx), gj = (j < 0 || j >= g.ny), gk = (k < 0 || k >= g.nz);
    const bool active = i <= g.nx && j <= g.ny && gi + gj + gk <= 1;
    const long long ge = active ? ghost_index(g, i, j, k) : 0;
    __nv_bfloat16* my_rows = rows[threadIdx.y] + threadIdx.x * 3 * mlp::RSTRIDE;
    const R* Gc = G + ge;  // variable c at Gc[c * GN + offset]
    float sc[NV];
    if (active) {
        const float rho = ld(Gc), E = ld(Gc + 4 * g.GN);
#pragma unroll
        for (int c = 0; c < NV; ++c) sc[c] = mlp::var_scale<float>(c, rho, E);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float x[mlp::NIN];
#pragma unroll
        for (int q = 0; q < mlp::NIN; ++q) x[q] = 0.0f;  // the row of an inactive lane is never read
        const int stp = d == 0 ? 1 : d == 1 ? g.gx : g.gx * g.gy;
        if (active) {
            float s5[NV][5];
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const R* p = Gc + (long long)c * g.GN;
#pragma unroll
                for (int o = 0; o < 5; ++o) s5[c][o] = ld(p + (o - 2) * stp);
            }
#pragma unroll
            for (int c = 0; c < NV; ++c) mlp::normalise5(s5[c], sc[c], x + c * 5);
        }
        mlp::stage_row(my_rows + d * mlp::RSTRIDE, x, true);
    }
    __syncwarp();  // the warp's rows staged
    mlp::warp_logits(wts, rows[threadIdx.y], lg[threadIdx.y]);
    __syncwarp();
    if (active) {
        const float* l3 = lg[threadIdx.y] + threadIdx.x * 3;
        flag[ext_index(g, i, j, k)] = fmaxf(l3[0], fmaxf(l3[1], l3[2])) > logit_thr ? 1 : 0;
    }
}

// The gate's flags widened to each cell's 3 x 3 x 3 neighbourhood (a cell is flagged when any cell
// around it is), for the cells the fused stage reconstructs.  Flags scored on a step's first stage
// and reused by its later stages then still cover a discontinuity that moves by less than a cell
// over the step (the CFL number bounds the wave speed x dt by the cell width).
__global__ void __launch_bounds__(128) k_gate_dilate(const unsigned char* __restrict__ f, unsigned char* __restrict__ o,
                                                     Geo g) {
    const int i = blockIdx.x * 128 + threadIdx.x, j = blockIdx.y, k = blockIdx.z;  // extended coordinates
    if (i >= g.ex) return;
    const int ey = g.ny + 2, ez = g.nz + 2;
    unsigned m = 0;
#pragma unroll
    for (int dk = -1; dk <= 1; ++dk) {
        const int kk = k + dk;
        if (kk < 0 || kk >= ez) continue;
#pragma unroll
        for (int dj = -1; dj <= 1; ++dj) {
            const int jj = j + dj;
            if (jj < 0 || jj >= ey) continue;
            const unsigned char* row = f + ((long long)kk * ey + jj) * g.ex;
            m |= __ldg(row + i);
            if (i > 0) m |= __ldg(row + i - 1);
            if (i + 1 < g.ex) m |= __ldg(row + i + 1);
        }
    }
    o[((long long)k * ey + j) * g.ex + i] = (unsigned char)m;
}

// LEARNED: the indicator gate of k_recon_learned, read from the flags k_gate wrote for this
// stage's input: flagged cells take CWENO4, the others R4, and a cell whose R4 traces break the
// floors is redone with CWENO4 (then first order with the positivity fallback)
template <bool LEARNED>
__global__ void __launch_bounds__(FS_NT, 1)
    k_stage_f32(const float* __restrict__ G, const double* U, const double* W, double* out, Geo g, int recon, int pad,
                double gamma, double r1_h, Stage st, DevScalars* __restrict__ ds, int slot,
                unsigned long long* __restrict__ counters, const unsigned char* __restrict__ gate = nullptr) {
    extern __shared__ float S[];  // traces [c][q][thread], then the -y face fluxes [c][thread]
    float* SFy = S + FS_NQ * FS_NT;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const float gm = (float)gamma, gm1 = (float)(gamma - 1.0);
    const long long tiles_x = fs_tiles_x(g.nx);
    const long long total = tiles_x * fs_tiles_y(g.ny) * g.nz;  // plane-units
    const long long b0 = (long long)blockIdx.x * total / gridDim.x, b1 = (long long)(blockIdx.x + 1) * total / gridDim.x;
    const double cdt = st.rhs_only ? 0.0 : st.c * ds->dt;
    const float r1h = (float)r1_h;
    float smax = 0.0f;
    unsigned nfall = 0, nflag = 0;
    for (long long pos = b0; pos < b1;) {
        const long long tile = pos / g.nz;
        const int kb = (int)(pos - tile * g.nz);
        const int ke = (int)min((long long)g.nz, kb + (b1 - pos));
        pos += ke - kb;
        const int i0 = (int)(tile % tiles_x) * FS_OX, j0 = (int)(tile / tiles_x) * FS_OY;
        const int i = i0 + lane - 1, j = j0 + w - 1;
        const int ihi = min(i0 + FS_OX, g.nx), jhi = min(j0 + FS_OY, g.ny);  // owned: [i0, ihi) x [j0, jhi)
        const bool own_x = i >= i0 && i < ihi, own_y = j >= j0 && j < jhi;
        const bool ring_x = (i == i0 - 1 || i == ihi), ring_y = (j == j0 - 1 || j == jhi);
        const bool owned = own_x && own_y;
        const bool ring = (ring_x && own_y) || (own_x && ring_y);
        // the gate's flag of the next plane, loaded a plane ahead (cells in [-1, n] along x and y)
        unsigned char fnext = 0;
        if (LEARNED && (owned || ring)) fnext = gate[ext_index(g, i, j, kb - 1)];
        float zp[NV][4];    // +z traces of the previous plane
        float Fzp[NV];      // flux of the previous plane's -z face
        float Pp[NV];       // x/y part of the previous plane's divergence
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            Fzp[c] = Pp[c] = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) zp[c][q] = 0.0f;
        }
#pragma unroll 1
        for (int k = kb - 1; k <= ke; ++k) {
            const bool edge = (k == kb - 1) || (k == ke);  // only the z traces of owned columns are used
            const bool active = owned || (ring && !edge);
            const long long ge = active ? ghost_index(g, i, j, k) : 0;
            bool full = false;
            if constexpr (LEARNED) {
                full = active && fnext != 0;
                if (full && owned && !edge) ++nflag;
                if ((owned || ring) && k < ke) fnext = gate[ext_index(g, i, j, k + 1)];
            }
            // the plane after the next one's stencils' last, into L2 while this plane is computed
            if (owned || ring) {
                const float* ahead = G + ghost_index(g, i, j, k) + (k + 3 < g.nz + GW ? 3 : 2) * (long long)(g.gx * g.gy);
#pragma unroll
                for (int c = 0; c < NV; ++c) prefetch_l2(ahead + (long long)c * g.GN);
            }
            // ---- reconstruction: all 24 traces of each variable into the shared array
            if (active) {
                const bool weno = !LEARNED && recon == HYPE_RECON_WENO3;
                bool linear = LEARNED ? !full : recon == HYPE_RECON_LINEAR4;
                bool ok = true;
                // one copy of the reconstruction in the code: with the gate, R4 traces that break
                // the floors are redone with CWENO4 on a second pass
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass) {
                    fs_recon_cell(S, G, g, ge, t, linear, weno);
                    ok = (LEARNED || pad) ? fs_admissible(S, t, gm1) : true;
                    if (!LEARNED || ok || !linear) break;
                    linear = false;
                }
                // positivity fallback: first order when the traces still break the floors
                if (!ok && pad) {
#pragma unroll 1
                    for (int c = 0; c < NV; ++c) {
                        const float v = __ldg(G + (long long)c * g.GN + ge);
                        for (int q = 0; q < NTR; ++q) S[(c * NTR + q) * FS_NT + t] = v;
                    }
                    if (owned && !edge) ++nfall;
                }
            }
            __syncthreads();
            // ---- Rusanov fluxes of the owned cells' faces: -x (the ring lane at the high side gives
            // the last cell's +x; the +x flux of every cell comes from its right neighbour lane by a
            // shuffle), -y and +y (each y face is solved by both of its cells: no exchange between
            // warps), -z (low side from registers)
            const bool plane = (k >= kb) && (k < ke);
            // z face first: it completes the previous plane (its stage value), then frees zp
            if (k >= kb && owned) {
                float Fz[NV];
                bool b = false;
                fs_face(S, t, t, 0, 16, zp, gm, gm1, Fz, smax, b, 2);  // L: registers (zl), R: own -z (q 16..19)
                if (b) fs_bad(ds, g, i, j, k);
                if (k > kb) {
                    const long long cell = ((long long)(k - 1) * g.ny + j) * g.nx + i;
#pragma unroll
                    for (int c = 0; c < NV; ++c) {
                        const double L = df_f2d(div_z_f(Pp[c], Fz[c] - Fzp[c], r1h));
                        const double u = (!st.rhs_only && st.a != 0.0) ? U[c * g.N + cell] : 0.0;
                        const double wv = st.rhs_only ? 0.0 : W[c * g.N + cell];
                        out[c * g.N + cell] = stage_value(st, cdt, u, wv, L);
                    }
                }
#pragma unroll
                for (int c = 0; c < NV; ++c) Fzp[c] = Fz[c];
            }
            if (owned && k < ke) {
#pragma unroll
                for (int c = 0; c < NV; ++c)
#pragma unroll
                    for (int q = 0; q < 4; ++q) zp[c][q] = S[(c * NTR + 20 + q) * FS_NT + t];
            }
            // x faces: every lane its -x face (the ring lane at the high side gives the last cell's +x),
            // the +x flux from the right neighbour lane
            float dF[NV];
            {
                float Fxl[NV];
#pragma unroll
                for (int c = 0; c < NV; ++c) Fxl[c] = 0.0f;
                if (plane && own_y && (own_x || i == ihi)) {
                    bool b = false;
                    fs_face(S, t - 1, t, 4, 0, nullptr, gm, gm1, Fxl, smax, b, 0);
                    if (b) fs_bad(ds, g, i, j, k);
                }
#pragma unroll
                for (int c = 0; c < NV; ++c) dF[c] = __shfl_down_sync(0xffffffffu, Fxl[c], 1) - Fxl[c];
            }
            // y faces: each owned cell and the ring row at the high side its -y face, shared through
            // the flux array (the row above gives each owned cell its +y face)
            float Fyl[NV];
            if (plane && own_x && (own_y || j == jhi)) {
                bool b = false;
                fs_face(S, t - 32, t, 12, 8, nullptr, gm, gm1, Fyl, smax, b, 1);
                if (b) fs_bad(ds, g, i, j, k);
#pragma unroll
                for (int c = 0; c < NV; ++c) SFy[c * FS_NT + t] = Fyl[c];
            }
            __syncthreads();  // every trace read (the next plane may overwrite them), -y fluxes written
            if (plane && owned) {
#pragma unroll
                for (int c = 0; c < NV; ++c) Pp[c] = div_xy_f(dF[c], SFy[c * FS_NT + t + 32] - Fyl[c], r1h);
            }
            // the flux array is next written after the next plane's first barrier, when every
            // thread has read it
        }
    }
    if (nfall) atomicAdd(&counters[1], (unsigned long long)nfall);
    if (LEARNED && nflag) atomicAdd(&counters[0], (unsigned long long)nflag);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    if (lane == 0 && smax > 0.0f) atomic_max_pos(&ds->smax_bits[slot], (double)smax);
}

// the stage combination alone, from an RHS already in L (the first stage of a step whose dt
// comes from that stage's own RHS): the same explicitly rounded value as the fused kernel's
__global__ void __launch_bounds__(256) k_stage_combine(const double* U, const double* W, const double* __restrict__ L,
                                                       double* out, long long n, Stage st,
                                                       const DevScalars* __restrict__ ds) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= n) return;
    const double cdt = st.rhs_only ? 0.0 : st.c * ds->dt;
    const double u = (!st.rhs_only && st.a != 0.0) ? U[q] : 0.0;
    const double w = st.rhs_only ? 0.0 : W[q];
    out[q] = stage_value(st, cdt, u, w, L[q]);
}

// dt from the largest wave speed, rounded as each reference program does:
// (1/3) (CFL h) / s_max (3d/weno4/Navier-Stokes-3D/rhs_function.c:438-440) or
// (CFL h) / (3 s_max) (3d/weno3/Euler/rhs_function.c:383)
// and, with viscosity, (1/3) (CFL h) / (s_max + 2 s_visc / h) (Navier-Stokes-3D/rhs_function.c:438)
__host__ __device__ inline double cfl_dt(double cfl_h, double smax, int recon, double smaxv = 0.0, double r1_h = 0.0,
                                         bool visc = false) {
    if (visc) return (1.0 / 3.0) * cfl_h / (smax + (r1_h * smaxv) * 2.0);
    return recon == HYPE_RECON_WENO3 ? cfl_h / (3.0 * smax) : (1.0 / 3.0) * cfl_h / (smax + 0.0);
}

// dt of the coming step and the time update (one thread)
__global__ void k_begin_step(DevScalars* ds, int dt_mode, int src_slot, int use_src, int reset_stages, double cfl_h,
                             int recon, double r1_h, int visc) {
    if (use_src && dt_mode != HYPE_DT_FIXED) {
        const double smax = __longlong_as_double((long long)ds->smax_bits[src_slot]);
        const double smaxv = __longlong_as_double((long long)ds->smaxv_bits[src_slot]);
        ds->dt = cfl_dt(cfl_h, smax, recon, smaxv, r1_h, visc != 0);
    }
    if (reset_stages)
        for (int s = 0; s < 4; ++s) ds->smax_bits[s] = ds->smaxv_bits[s] = 0ull;
    ds->t += ds->dt;
}

// sum |a - b| and sum |b| over n values (two doubles accumulated with atomics)
__global__ void k_l1(const double* __restrict__ a, const double* __restrict__ b, long long n, double* __restrict__ acc) {
    double d = 0.0, r = 0.0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        d += fabs(a[q] - b[q]);
        r += fabs(b[q]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        d += __shfl_xor_sync(0xffffffffu, d, o);
        r += __shfl_xor_sync(0xffffffffu, r, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&acc[0], d);
        atomicAdd(&acc[1], r);
    }
}

__global__ void k_reset_slot(DevScalars* ds, int slot) {
    ds->smax_bits[slot] = 0ull;
    ds->smaxv_bits[slot] = 0ull;
    ds->bad = ~0ull;
}

// AoS [cell][c] <-> SoA [c][cell]
__global__ void k_aos_to_soa(const double* __restrict__ a, double* __restrict__ s, long long N) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= N * NV) return;
    const long long cell = q / NV;
    const int c = (int)(q - cell * NV);
    s[c * N + cell] = a[q];
}
__global__ void k_soa_to_aos(const double* __restrict__ s, double* __restrict__ a, long long N) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= N * NV) return;
    const long long cell = q / NV;
    const int c = (int)(q - cell * NV);
    a[q] = s[c * N + cell];
}

// ---------------------------------------------------------------- monitor diagnostics
// KineticEnergy (3d/weno4/Navier-Stokes-3D/kinetic_energy.c:11-44): sum of
// h^3 (|rho u|^2 / 2 rho); Dissipation (dissipation.c:11-67): sum over cells of
// tau : grad v with central velocity differences and the Stokes stress of viscosity
// mu.  Neighbours across a non-periodic face are the context's ghost values of the
// state.  Deterministic: one partial pair per block, then one block sums the
// partials in a fixed order.
constexpr int kMonThreads = 256;

__device__ __forceinline__ void block_sum2(double& a, double& b, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        sh[2 * w] = a;
        sh[2 * w + 1] = b;
    }
    __syncthreads();
    if (w == 0) {
        a = l < (int)(blockDim.x >> 5) ? sh[2 * l] : 0.0;
        b = l < (int)(blockDim.x >> 5) ? sh[2 * l + 1] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
    }
}

__device__ __forceinline__ void vel_at(const double* __restrict__ U, const Geo& g, int i, int j, int k, double* v) {
    int fi = 0, fj = 0, fk = 0;
    const int mi = bmap(i, g.nx, g.bc[0], g.bc[1], &fi);
    const int mj = bmap(j, g.ny, g.bc[2], g.bc[3], &fj);
    const int mk = bmap(k, g.nz, g.bc[4], g.bc[5], &fk);
    const long long q = ((long long)mk * g.ny + mj) * g.nx + mi;
    const double rho = __ldg(U + q);
    v[0] = (fi ? -1.0 : 1.0) * __ldg(U + g.N + q) / rho;
    v[1] = (fj ? -1.0 : 1.0) * __ldg(U + 2 * g.N + q) / rho;
    v[2] = (fk ? -1.0 : 1.0) * __ldg(U + 3 * g.N + q) / rho;
}

__global__ void __launch_bounds__(kMonThreads) k_monitor(const double* __restrict__ U, Geo g, double vol, double r1_2h,
                                                         double mu, double* __restrict__ part) {
    __shared__ double sh[2 * (kMonThreads / 32)];
    double ke = 0.0, dr = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < g.N; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % g.nx), j = (int)((q / g.nx) % g.ny), k = (int)(q / ((long long)g.nx * g.ny));
        const double rho = __ldg(U + q), mx = __ldg(U + g.N + q), my = __ldg(U + 2 * g.N + q), mz = __ldg(U + 3 * g.N + q);
        ke += vol * 0.5 * (mx * mx + my * my + mz * mz) / rho;
        double a[3], b[3], vg[3][3];  // vg[a][b]: d(velocity a)/d(x_b)
        vel_at(U, g, i + 1, j, k, a);
        vel_at(U, g, i - 1, j, k, b);
#pragma unroll
        for (int c = 0; c < 3; ++c) vg[c][0] = r1_2h * (a[c] - b[c]);
        vel_at(U, g, i, j + 1, k, a);
        vel_at(U, g, i, j - 1, k, b);
#pragma unroll
        for (int c = 0; c < 3; ++c) vg[c][1] = r1_2h * (a[c] - b[c]);
        vel_at(U, g, i, j, k + 1, a);
        vel_at(U, g, i, j, k - 1, b);
#pragma unroll
        for (int c = 0; c < 3; ++c) vg[c][2] = r1_2h * (a[c] - b[c]);
        const double div_v = -(2.0 / 3.0) * mu * (vg[0][0] + vg[1][1] + vg[2][2]);
        const double txx = div_v + 2.0 * mu * vg[0][0], txy = mu * (vg[0][1] + vg[1][0]), txz = mu * (vg[0][2] + vg[2][0]);
        const double tyy = div_v + 2.0 * mu * vg[1][1], tyz = mu * (vg[1][2] + vg[2][1]), tzz = div_v + 2.0 * mu * vg[2][2];
        dr += (txx * vg[0][0] + txy * vg[0][1] + txz * vg[0][2]) + (txy * vg[1][0] + tyy * vg[1][1] + tyz * vg[1][2]) +
              (txz * vg[2][0] + tyz * vg[2][1] + tzz * vg[2][2]);
    }
    block_sum2(ke, dr, sh);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = ke;
        part[2 * blockIdx.x + 1] = dr;
    }
}

__global__ void __launch_bounds__(kMonThreads) k_monitor_sum(const double* __restrict__ part, int nblk, double* out) {
    __shared__ double sh[2 * (kMonThreads / 32)];
    double ke = 0.0, dr = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        ke += part[2 * b];
        dr += part[2 * b + 1];
    }
    block_sum2(ke, dr, sh);
    if (threadIdx.x == 0) {
        out[0] = ke;
        out[1] = dr;
    }
}

}  // namespace euler
}  // namespace hype

using namespace hype;
using namespace hype::euler;

static inline double bits_to_double(unsigned long long b) {
    double d;
    memcpy(&d, &b, sizeof(d));
    return d;
}

struct hype_euler {
    hype_euler_params p;
    Geo g;
    cudaStream_t stream = nullptr;
    double* U = nullptr;   // resident state (SoA)
    double* W = nullptr;   // stage state
    double* L = nullptr;   // RHS buffer (rhs-only calls)
    double* S = nullptr;   // scratch SoA state for host RHS calls
    void* T = nullptr;     // traces
    double* Fx = nullptr;
    double* Fy = nullptr;
    double* Fz = nullptr;
    double* stage_aos = nullptr;  // device AoS staging
    void* G = nullptr;            // ghosted stage input in the reconstruction's precision
    double* C4 = nullptr;         // viscous runs: R4 coefficients [5][20][ext cells] for the face gradients
    double* mon = nullptr;        // monitor partial sums (2 per block) and the result pair
    DevScalars* ds = nullptr;
    DevScalars* hs = nullptr;  // pinned host copy
    double* pin = nullptr;     // pinned host staging for AoS transfers
    // learned indicator: BF16 parameters, logit threshold, counters (flagged, positivity fallbacks)
    mlp::MmaWeights* mlp = nullptr;  // packed for the tensor-core inference
    // fused FP32 stage: the gate's flags (one byte per extended cell) and, when the gate is scored
    // once per step, their one-cell widening that the step's stages read
    unsigned char* gate = nullptr;
    unsigned char* gate_wide = nullptr;
    // the gated FP64 reconstruction: flags, and a bound of each variable's polynomial, per extended cell
    unsigned char* flag64 = nullptr;
    float* bound64 = nullptr;
    int gate_per_step = 0;
    float logit_thr = 0.0f;
    unsigned long long* mlp_cnt = nullptr;
    // per-kernel event timing inside a timed region (hype_euler_profile)
    bool prof = false;
    // the steady-state step (every step after the first of a call) captured as a CUDA graph,
    // with the launch choices it was captured under and the kernels it launches
    cudaGraphExec_t step_graph = nullptr;
    long long graph_key[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    long long graph_launches = 0;
    // stage kernels: HYPE_STAGE_AUTO takes the fused FP32 stage where it applies; the unfused
    // kernels' trace and face-flux buffers are allocated when first needed
    int stage_mode = HYPE_STAGE_AUTO;
    int nsm = 1;
    double* acc = nullptr;  // two doubles: k_l1's sums
    std::vector<cudaEvent_t> ev;  // pairs (start, end)
    std::vector<int> ev_kind;     // 0 recon, 1 faces (3 directions), 2 update
    size_t ev_used = 0;
};

static void prof_mark(hype_euler* e, int kind, bool start) {
    if (!e->prof) return;
    if (start) {
        if (e->ev_used + 2 > e->ev.size()) {
            for (int q = 0; q < 64; ++q) {
                cudaEvent_t x;
                cudaEventCreate(&x);
                e->ev.push_back(x);
            }
            e->ev_kind.resize(e->ev.size() / 2);
        }
        e->ev_kind[e->ev_used / 2] = kind;
        cudaEventRecord(e->ev[e->ev_used], e->stream);
    } else {
        cudaEventRecord(e->ev[e->ev_used + 1], e->stream);
        e->ev_used += 2;
    }
}

// the face-flux launches of one RHS (FP32 or FP64 traces), for the context's flux; vp: with viscosity
template <int FLUX>
static int launch_faces_t(const Geo& g, const void* T, double* Fx, double* Fy, double* Fz, double gamma, DevScalars* ds,
                          int slot, bool f32, cudaStream_t st, const double* C4, const Visc* vp) {
    if (f32) {
        const dim3 bf(32, 4);
        const dim3 gx(cdiv(g.nx + 1, 32), cdiv(g.ny, 4), g.nz), gy(cdiv(g.nx, 32), cdiv(g.ny + 1, 4), g.nz),
            gz(cdiv(g.nx, 32), cdiv(g.ny, 4), g.nz + 1);
        k_faces_f32<0, FLUX><<<gx, bf, 0, st>>>((const float*)T, Fx, g, gamma, ds, slot);
        k_faces_f32<1, FLUX><<<gy, bf, 0, st>>>((const float*)T, Fy, g, gamma, ds, slot);
        k_faces_f32<2, FLUX><<<gz, bf, 0, st>>>((const float*)T, Fz, g, gamma, ds, slot);
        return 3;
    }
    const long long most = std::max({(long long)(g.nx + 1) * g.ny * g.nz, (long long)g.nx * (g.ny + 1) * g.nz,
                                     (long long)g.nx * g.ny * (g.nz + 1)});
    if (vp) k_faces_visc64<FLUX><<<dim3(cdiv(most, 32), 3), 128, 0, st>>>((const double*)T, Fx, Fy, Fz, g, gamma, ds, slot, C4, *vp);
    else k_faces64<FLUX><<<dim3(cdiv(most, 32), 3), 128, 0, st>>>((const double*)T, Fx, Fy, Fz, g, gamma, ds, slot);
    return 1;
}

static int launch_faces(const Geo& g, const void* T, double* Fx, double* Fy, double* Fz, double gamma, DevScalars* ds,
                        int slot, bool f32, int flux, cudaStream_t st, const double* C4 = nullptr, const Visc* vp = nullptr) {
    const auto go = flux == HYPE_FLUX_HLLC      ? launch_faces_t<HYPE_FLUX_HLLC>
                    : flux == HYPE_FLUX_ROTHLLC ? launch_faces_t<HYPE_FLUX_ROTHLLC>
                                                : launch_faces_t<HYPE_FLUX_RUSANOV>;
    return go(g, T, Fx, Fy, Fz, gamma, ds, slot, f32, st, C4, vp);
}

static int launch_rhs(hype_euler* e, const double* Win, int slot) {
    const Geo& g = e->g;
    const dim3 br(32, 4), gr(cdiv(g.nx + 2, 32), cdiv(g.ny + 2, 4), g.nz + 2);
    const bool f32 = e->p.precision == HYPE_PREC_FP32;
    // HYPE_PREC_DF64 asks for FP64's error bars on the FP32 pipe, which pairs of FP32 numbers gave.  The FP64 kernels'
    // integer form is closer to 64 bits and faster, and serves both (two steps, pairs against this: 16^3 707 -> 300
    // us, 161 x 150 x 143 47.6 -> 43.4 ms, Navier-Stokes 96^3 40.3 -> 31.9, blast 96^3 with the fallback 21.5 -> 15.2).
    const int rec = e->p.recon;
    prof_mark(e, 0, true);
    if (f32) k_ghost<float><<<ghost_grid(g), kGhostThreads, 0, e->stream>>>(Win, (float*)e->G, g);
    else k_ghost<double><<<ghost_grid(g), kGhostThreads, 0, e->stream>>>(Win, (double*)e->G, g);
    HYPE_LAUNCHED(1);
    const double gm1 = e->p.gamma - 1.0;
    const size_t ck_bytes = (f32 && e->p.positivity) ? sizeof(float) * 4 * 2 * NTR * 32 : 0;
    if (e->p.recon == HYPE_RECON_LEARNED) {
        if (!e->mlp) return HYPE_ERR_ARG;  // hype_euler_set_mlp first
        if (f32)
            k_recon_learned<<<gr, br, 0, e->stream>>>((const float*)e->G, (float*)e->T, g, e->mlp, e->logit_thr, gm1,
                                                      e->p.positivity, e->mlp_cnt);
        else {
            const double* G = (const double*)e->G;
            double* T = (double*)e->T;
            k_gate<double><<<gr, br, 0, e->stream>>>(G, e->flag64, g, e->mlp, e->logit_thr);
            k_recon64<HYPE_RECON_LEARNED, false><<<dim3(cdiv(g.NE, kReconThreads), NV), kReconThreads, 0, e->stream>>>(
                G, T, g, gm1, e->mlp_cnt, nullptr, e->flag64, e->bound64);
            k_gated_check<<<cdiv(g.NE, kGatedThreads), kGatedThreads, 0, e->stream>>>(G, T, g, gm1, e->p.positivity, e->flag64,
                                                                                     e->bound64, e->mlp_cnt);
            HYPE_LAUNCHED(2);
        }
    } else if (f32) {
        k_recon_f32<<<gr, br, ck_bytes, e->stream>>>((const float*)e->G, (float*)e->T, g, rec, e->p.positivity, gm1,
                                                     e->mlp_cnt);
    } else {
        launch_recon64(g, (const double*)e->G, (double*)e->T, rec, e->p.positivity, gm1, e->mlp_cnt, e->C4, e->stream);
    }
    int nk = 2;
    prof_mark(e, 0, false);
    prof_mark(e, 1, true);
    if (e->C4) {
        // Navier-Stokes: the inviscid flux plus the average of both sides' viscous fluxes
        const double mu = e->p.mu, g = e->p.gamma;
        const Visc vp{mu, e->p.cv * mu * g / e->p.prandtl, std::max((4. / 3.) * mu, g * mu / e->p.prandtl), 1.0 / e->p.h};
        nk += launch_faces(e->g, e->T, e->Fx, e->Fy, e->Fz, e->p.gamma, e->ds, slot, false, e->p.flux, e->stream, e->C4, &vp);
    } else {
        nk += launch_faces(e->g, e->T, e->Fx, e->Fy, e->Fz, e->p.gamma, e->ds, slot, f32, e->p.flux, e->stream);
    }
    prof_mark(e, 1, false);
    HYPE_LAUNCHED(nk - 1);  // the ghost fill is counted above
    return HYPE_OK;
}

static int launch_update(hype_euler* e, const double* U, const double* W, double* out, Stage st) {
    const Geo& g = e->g;
    const unsigned b = kUpdateThreads;
    const dim3 gr = update_grid(g);
    prof_mark(e, 2, true);
    if (e->p.precision == HYPE_PREC_FP32)
        k_update<true><<<gr, b, 0, e->stream>>>(e->Fx, e->Fy, e->Fz, U, W, out, g, 1.0 / e->p.h, st, e->ds);
    else
        k_update<false><<<gr, b, 0, e->stream>>>(e->Fx, e->Fy, e->Fz, U, W, out, g, 1.0 / e->p.h, st, e->ds);
    prof_mark(e, 2, false);
    HYPE_LAUNCHED(1);
    return HYPE_OK;
}

// whether the context's current options run the fused FP32 stage kernel
static bool uses_fused(const hype_euler* e) {
    return e->stage_mode == HYPE_STAGE_AUTO && e->p.precision == HYPE_PREC_FP32 && e->p.flux == HYPE_FLUX_RUSANOV &&
           !e->C4 && (e->p.recon == HYPE_RECON_CWENO4 || e->p.recon == HYPE_RECON_LINEAR4 ||
                      e->p.recon == HYPE_RECON_WENO3 || (e->p.recon == HYPE_RECON_LEARNED && e->mlp && e->gate));
}

// the unfused kernels' face traces and face fluxes, allocated on first use (never inside a
// stream capture: every entry point that may launch them calls this first)
static int ensure_unfused(hype_euler* e) {
    if (e->T) return HYPE_OK;
    const Geo& g = e->g;
    const hype_euler_params* p = &e->p;
    const size_t tsz = (p->precision == HYPE_PREC_FP32 ? sizeof(float) : sizeof(double)) * NV * NTR * (size_t)g.NE;
    cudaError_t ce = cudaMalloc(&e->T, tsz);
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&e->Fx, sizeof(double) * NV * (size_t)(p->nx + 1) * p->ny * p->nz);
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&e->Fy, sizeof(double) * NV * (size_t)p->nx * (p->ny + 1) * p->nz);
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&e->Fz, sizeof(double) * NV * (size_t)p->nx * p->ny * (p->nz + 1));
    if (ce != cudaSuccess) {
        cudaFree(e->T); cudaFree(e->Fx); cudaFree(e->Fy); cudaFree(e->Fz);
        e->T = nullptr; e->Fx = e->Fy = e->Fz = nullptr;
        set_last_error("cudaMalloc (face traces)", ce);
        return HYPE_ERR_NOMEM;
    }
    return HYPE_OK;
}

static int prepare(hype_euler* e) { return uses_fused(e) ? HYPE_OK : ensure_unfused(e); }

// One RK stage: out = a U + b W + (c dt) L(Win) (or out = L(Win) for RHS-only calls), with the
// wave-speed maximum into slot.  The fused FP32 stage is the device ghost fill plus one kernel;
// every other form is ghost fill, reconstruction, three face-flux kernels and the update.
static int launch_stage(hype_euler* e, const double* Win, const double* U, const double* W, double* out, Stage st,
                        int slot) {
    if (!uses_fused(e)) {
        int rc = launch_rhs(e, Win, slot);
        if (rc) return rc;
        return launch_update(e, U, W, out, st);
    }
    const Geo& g = e->g;
    prof_mark(e, 0, true);
    k_ghost<float><<<ghost_grid(g), kGhostThreads, 0, e->stream>>>(Win, (float*)e->G, g);
    const bool learned = e->p.recon == HYPE_RECON_LEARNED;
    // the gate's flags for this stage's input; scored once per step, on the first stage's input
    // (slot 0) and for RHS-only calls (slot 4), then widened by a cell for the step's later stages
    const bool score = learned && (!e->gate_per_step || slot == 0 || slot == 4);
    if (score) {
        const dim3 br(32, 4), gr(cdiv(g.nx + 2, 32), cdiv(g.ny + 2, 4), g.nz + 2);
        k_gate<float><<<gr, br, 0, e->stream>>>((const float*)e->G, e->gate, g, e->mlp, e->logit_thr);
        if (e->gate_per_step)
            k_gate_dilate<<<dim3(cdiv(g.ex, 128), g.ny + 2, g.nz + 2), 128, 0, e->stream>>>(e->gate, e->gate_wide, g);
    }
    prof_mark(e, 0, false);
    prof_mark(e, 1, true);
    const long long units = fs_tiles_x(g.nx) * fs_tiles_y(g.ny) * g.nz;
    const unsigned blocks = (unsigned)std::min<long long>(e->nsm, units);
    if (learned)
        k_stage_f32<true><<<blocks, FS_NT, FS_SMEM, e->stream>>>((const float*)e->G, U, W, out, g, e->p.recon,
                                                                e->p.positivity, e->p.gamma, 1.0 / e->p.h, st, e->ds,
                                                                slot, e->mlp_cnt,
                                                                e->gate_per_step ? e->gate_wide : e->gate);
    else
        k_stage_f32<false><<<blocks, FS_NT, FS_SMEM, e->stream>>>((const float*)e->G, U, W, out, g, e->p.recon,
                                                                 e->p.positivity, e->p.gamma, 1.0 / e->p.h, st, e->ds,
                                                                 slot, e->mlp_cnt);
    prof_mark(e, 1, false);
    HYPE_LAUNCHED(2 + (score ? 1 + (e->gate_per_step ? 1 : 0) : 0));
    return HYPE_OK;
}

// the first stage of a step whose dt comes from that stage's own RHS: RHS into L, dt, then the
// stage combination (fused form) or the update kernel (unfused)
static int launch_first_stage_from_rhs(hype_euler* e, int mode, double cfl_h, Stage s12) {
    int rc;
    if (uses_fused(e)) {
        const Stage rhs{0.0, 0.0, 0.0, 1};
        if ((rc = launch_stage(e, e->U, nullptr, nullptr, e->L, rhs, 0))) return rc;
    } else if ((rc = launch_rhs(e, e->U, 0))) {
        return rc;
    }
    k_begin_step<<<1, 1, 0, e->stream>>>(e->ds, mode, 0, 1, 0, cfl_h, e->p.recon, 1.0 / e->p.h, e->C4 != nullptr);
    HYPE_LAUNCHED(1);
    if (!uses_fused(e)) return launch_update(e, e->U, e->U, e->W, s12);
    const long long n = NV * e->g.N;
    prof_mark(e, 2, true);
    k_stage_combine<<<cdiv(n, 256), 256, 0, e->stream>>>(e->U, e->U, e->L, e->W, n, s12, e->ds);
    prof_mark(e, 2, false);
    HYPE_LAUNCHED(1);
    return HYPE_OK;
}

extern "C" int hype_euler_create(const hype_euler_params* p, hype_euler** out) {
    if (!p || !out) return HYPE_ERR_ARG;
    *out = nullptr;
    if (p->nx < 3 || p->ny < 3 || p->nz < 3 || !(p->h > 0) || !(p->cfl > 0) || !(p->gamma > 1.0)) return HYPE_ERR_ARG;
    for (int f = 0; f < 6; ++f)
        if (p->bc[f] < HYPE_BC_PERIODIC || p->bc[f] > HYPE_BC_TRANSMISSIVE) return HYPE_ERR_ARG;
    for (int d = 0; d < 3; ++d)
        if ((p->bc[2 * d] == HYPE_BC_PERIODIC) != (p->bc[2 * d + 1] == HYPE_BC_PERIODIC)) return HYPE_ERR_ARG;
    if (p->recon < HYPE_RECON_CWENO4 || p->recon > HYPE_RECON_WENO3) return HYPE_ERR_ARG;
    if (p->precision != HYPE_PREC_FP64 && p->precision != HYPE_PREC_FP32 && p->precision != HYPE_PREC_DF64)
        return HYPE_ERR_ARG;
    // HYPE_PREC_DF64 has not taken WENO3, nor viscosity with the HLLC family, since it had kernels of its own; callers
    // rely on the refusals
    if (p->precision == HYPE_PREC_DF64 && p->recon == HYPE_RECON_WENO3) return HYPE_ERR_UNSUPPORTED;
    if (p->dt_mode < HYPE_DT_MONITOR || p->dt_mode > HYPE_DT_FIXED) return HYPE_ERR_ARG;
    if (p->flux < HYPE_FLUX_RUSANOV || p->flux > HYPE_FLUX_ROTHLLC) return HYPE_ERR_ARG;
    if (p->positivity != 0 && p->positivity != 1) return HYPE_ERR_ARG;
    // viscosity: in FP64 or HYPE_PREC_DF64, with the CWENO4, R4 or WENO3 traces; the gradients always come from R4
    const bool visc = p->mu != 0.0;
    if (visc && (!(p->mu > 0.0) || !(p->prandtl > 0.0) || !(p->cv > 0.0) || p->precision == HYPE_PREC_FP32 ||
                 p->recon == HYPE_RECON_LEARNED))
        return HYPE_ERR_ARG;
    if (visc && p->precision == HYPE_PREC_DF64 && p->flux != HYPE_FLUX_RUSANOV) return HYPE_ERR_UNSUPPORTED;
    hype_euler* e = new hype_euler();
    e->p = *p;
    Geo& g = e->g;
    g.nx = p->nx; g.ny = p->ny; g.nz = p->nz;
    for (int f = 0; f < 6; ++f) g.bc[f] = p->bc[f];
    g.N = (long long)p->nx * p->ny * p->nz;
    g.NE = (long long)(p->nx + 2) * (p->ny + 2) * (p->nz + 2);
    g.ex = p->nx + 2;
    g.ey = p->ny + 2;
    set_ghost_extents(g);
    const size_t sN = sizeof(double) * NV * (size_t)g.N;
    int rc = HYPE_OK;
    auto fail = [&](int code) {
        hype_euler_destroy(e);
        return code;
    };
    cudaError_t ce;
#define ALLOC(ptr, bytes)                                  \
    ce = cudaMalloc((void**)&(ptr), (bytes));              \
    if (ce != cudaSuccess) {                               \
        set_last_error("cudaMalloc", ce);                  \
        return fail(HYPE_ERR_NOMEM);                       \
    }
    ce = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
    if (ce != cudaSuccess) {
        set_last_error("cudaStreamCreate", ce);
        return fail(HYPE_ERR_CUDA);
    }
    ALLOC(e->U, sN);
    ALLOC(e->W, sN);
    ALLOC(e->L, sN);
    ALLOC(e->S, sN);
    ALLOC(e->stage_aos, sN);
    ALLOC(e->acc, 2 * sizeof(double));
    ALLOC(e->ds, sizeof(DevScalars));
    ALLOC(e->mlp_cnt, 2 * sizeof(unsigned long long));
    ALLOC(e->G, (p->precision == HYPE_PREC_FP32 ? sizeof(float) : sizeof(double)) * NV * (size_t)g.GN);
    if (visc) ALLOC(e->C4, sizeof(double) * NV * 20 * (size_t)g.NE);
#undef ALLOC
    {
        int dev = 0;
        ce = cudaGetDevice(&dev);
        if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&e->nsm, cudaDevAttrMultiProcessorCount, dev);
        if (ce == cudaSuccess)
            ce = cudaFuncSetAttribute(k_stage_f32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM);
        if (ce == cudaSuccess)
            ce = cudaFuncSetAttribute(k_stage_f32<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM);
        if (ce != cudaSuccess) {
            set_last_error("hype_euler_create (device attributes)", ce);
            return fail(HYPE_ERR_CUDA);
        }
        // the FP32 Rusanov form runs fused (the learned gate too, once its network is set): no trace
        // buffers up front; every other form allocates them now
        const bool fusable = p->precision == HYPE_PREC_FP32 && p->flux == HYPE_FLUX_RUSANOV && !visc;
        if (!fusable && (rc = prepare(e))) return fail(rc);
    }
    ce = cudaMemset(e->mlp_cnt, 0, 2 * sizeof(unsigned long long));
    if (ce != cudaSuccess) {
        set_last_error("cudaMemset", ce);
        return fail(HYPE_ERR_CUDA);
    }
    ce = cudaMallocHost((void**)&e->hs, sizeof(DevScalars));
    if (ce != cudaSuccess) {
        set_last_error("cudaMallocHost", ce);
        return fail(HYPE_ERR_NOMEM);
    }
    DevScalars z;
    memset(&z, 0, sizeof(z));
    z.bad = ~0ull;
    ce = cudaMemcpy(e->ds, &z, sizeof(z), cudaMemcpyHostToDevice);
    if (ce != cudaSuccess) {
        set_last_error("cudaMemcpy", ce);
        return fail(HYPE_ERR_CUDA);
    }
    *out = e;
    return rc;
}

extern "C" void hype_euler_destroy(hype_euler* e) {
    if (!e) return;
    if (e->stream) cudaStreamSynchronize(e->stream);
    cudaFree(e->U); cudaFree(e->W); cudaFree(e->L); cudaFree(e->S); cudaFree(e->T);
    if (e->bound64 != (float*)e->stage_aos) cudaFree(e->bound64);
    cudaFree(e->Fx); cudaFree(e->Fy); cudaFree(e->Fz); cudaFree(e->stage_aos); cudaFree(e->ds); cudaFree(e->G);
    cudaFree(e->mlp); cudaFree(e->gate); cudaFree(e->gate_wide); cudaFree(e->flag64); cudaFree(e->mlp_cnt); cudaFree(e->C4); cudaFree(e->mon); cudaFree(e->acc);
    if (e->hs) cudaFreeHost(e->hs);
    for (auto x : e->ev) cudaEventDestroy(x);
    if (e->step_graph) cudaGraphExecDestroy(e->step_graph);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
}

static int h2d_aos(hype_euler* e, const double* aos, double* soa) {
    const long long n = e->g.N * NV;
    HYPE_CK(cudaMemcpyAsync(e->stage_aos, aos, sizeof(double) * n, cudaMemcpyHostToDevice, e->stream));
    k_aos_to_soa<<<cdiv(n, 256), 256, 0, e->stream>>>(e->stage_aos, soa, e->g.N);
    HYPE_LAUNCHED(1);
    return HYPE_OK;
}

static int d2h_aos(hype_euler* e, const double* soa, double* aos) {
    const long long n = e->g.N * NV;
    k_soa_to_aos<<<cdiv(n, 256), 256, 0, e->stream>>>(soa, e->stage_aos, e->g.N);
    HYPE_LAUNCHED(1);
    HYPE_CK(copy_to_host(aos, e->stage_aos, sizeof(double) * n, e->stream));
    return HYPE_OK;
}

static int read_scalars(hype_euler* e) {
    HYPE_CK(cudaMemcpyAsync(e->hs, e->ds, sizeof(DevScalars), cudaMemcpyDeviceToHost, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return HYPE_OK;
}

static int rhs_core(hype_euler* e, const double* dU, double* dRHS, double* dt_out) {
    int rc;
    if ((rc = prepare(e))) return rc;
    k_reset_slot<<<1, 1, 0, e->stream>>>(e->ds, 4);
    HYPE_LAUNCHED(1);
    Stage st{0.0, 0.0, 0.0, 1};
    if ((rc = launch_stage(e, dU, nullptr, nullptr, dRHS, st, 4))) return rc;
    if ((rc = read_scalars(e))) return rc;
    const double smax = bits_to_double(e->hs->smax_bits[4]);
    const double smaxv = bits_to_double(e->hs->smaxv_bits[4]);
    if (dt_out) *dt_out = cfl_dt(e->p.cfl * e->p.h, smax, e->p.recon, smaxv, 1.0 / e->p.h, e->C4 != nullptr);
    if (e->hs->bad != ~0ull) return HYPE_ERR_STATE;
    return HYPE_OK;
}

extern "C" int hype_euler_rhs(hype_euler* e, double t, const double* U_aos, double* RHS_aos, double* dt_out) {
    (void)t;  // the Euler RHS is autonomous
    if (!e || !U_aos || !RHS_aos) return HYPE_ERR_ARG;
    int rc;
    if ((rc = h2d_aos(e, U_aos, e->S))) return rc;
    rc = rhs_core(e, e->S, e->L, dt_out);
    if (rc && rc != HYPE_ERR_STATE) return rc;
    int rc2 = d2h_aos(e, e->L, RHS_aos);
    if (rc2) return rc2;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return rc;
}

extern "C" int hype_euler_rhs_device(hype_euler* e, double t, const double* dU, double* dRHS, double* dt_out) {
    (void)t;
    if (!e || !dU || !dRHS) return HYPE_ERR_ARG;
    return rhs_core(e, dU, dRHS, dt_out);
}

extern "C" int hype_euler_get_params(const hype_euler* e, hype_euler_params* out) {
    if (!e || !out) return HYPE_ERR_ARG;
    *out = e->p;
    return HYPE_OK;
}

extern "C" int hype_euler_upload(hype_euler* e, const double* U_aos) {
    if (!e || !U_aos) return HYPE_ERR_ARG;
    int rc = h2d_aos(e, U_aos, e->U);
    if (rc) return rc;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return HYPE_OK;
}

extern "C" int hype_euler_download(hype_euler* e, double* U_aos) {
    if (!e || !U_aos) return HYPE_ERR_ARG;
    int rc = d2h_aos(e, e->U, U_aos);
    if (rc) return rc;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return HYPE_OK;
}

extern "C" double* hype_euler_state_device(hype_euler* e) { return e ? e->U : nullptr; }

extern "C" int hype_euler_sync(hype_euler* e) {
    if (!e) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return HYPE_OK;
}

// One SSPRK(4,3) step after the first of a call: dt from the previous step (MONITOR) or as
// set, then the four stages (the device scalars carry everything that changes between steps)
static int launch_steady_step(hype_euler* e, int mode, double cfl_h) {
    const Stage s12{0.0, 1.0, 0.5, 0};
    const Stage s3{2.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0, 0};
    int rc;
    k_begin_step<<<1, 1, 0, e->stream>>>(e->ds, mode, 3, mode == HYPE_DT_MONITOR, 1, cfl_h, e->p.recon, 1.0 / e->p.h,
                                         e->C4 != nullptr);
    HYPE_LAUNCHED(1);
    if ((rc = launch_stage(e, e->U, e->U, e->U, e->W, s12, 0))) return rc;
    if ((rc = launch_stage(e, e->W, e->U, e->W, e->W, s12, 1))) return rc;
    if ((rc = launch_stage(e, e->W, e->U, e->W, e->W, s3, 2))) return rc;
    return launch_stage(e, e->W, e->U, e->W, e->U, s12, 3);
}

// The steady-state step as a CUDA graph (replayed instead of ~25 launches per step; what
// matters on small grids), recaptured when a launch choice changes; falls back to launching
// (returns false) while profiling or if the capture fails.
static bool steady_step_graph(hype_euler* e, int mode, double cfl_h) {
    if (e->prof) return false;
    long long lt;
    memcpy(&lt, &e->logit_thr, sizeof(float));
    const long long key[8] = {mode, e->p.recon, e->p.flux, e->p.precision,
                              e->p.positivity + 2 * e->stage_mode + 8 * e->gate_per_step,
                              (long long)(size_t)e->mlp, lt, (long long)(cfl_h * 1e15)};
    if (e->step_graph && memcmp(key, e->graph_key, sizeof(key)) == 0) return true;
    if (e->step_graph) {
        cudaGraphExecDestroy(e->step_graph);
        e->step_graph = nullptr;
    }
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const long long l0 = hype_launch_count();
    const int rc = launch_steady_step(e, mode, cfl_h);
    const cudaError_t ce = cudaStreamEndCapture(e->stream, &graph);
    const long long nl = hype_launch_count() - l0;
    count_launch(-nl);  // captured, not launched
    if (rc != HYPE_OK || ce != cudaSuccess || !graph) {
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        return false;
    }
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    e->step_graph = exec;
    memcpy(e->graph_key, key, sizeof(key));
    e->graph_launches = nl;
    return true;
}

extern "C" int hype_euler_step(hype_euler* e, int nsteps, double* t_inout, double* dt_inout, hype_status* st) {
    if (!e || nsteps < 0 || !t_inout || !dt_inout) return HYPE_ERR_ARG;
    const int mode = e->p.dt_mode;
    if (mode == HYPE_DT_FIXED && !(*dt_inout > 0)) return HYPE_ERR_ARG;
    const double cfl_h = e->p.cfl * e->p.h;
    int rc;
    if ((rc = prepare(e))) return rc;
    // host-side initial values of t, dt, flags
    DevScalars init;
    memset(&init, 0, sizeof(init));
    init.t = *t_inout;
    init.dt = *dt_inout;
    init.bad = ~0ull;
    HYPE_CK(cudaMemcpyAsync(e->ds, &init, sizeof(init), cudaMemcpyHostToDevice, e->stream));
    const bool first_from_rhs = (mode != HYPE_DT_FIXED) && !(*dt_inout > 0);
    // SSPRK(4,3) (PETSc TSSSP RKS3, 4 stages; Ketcheson 2008):
    //   u1 = u + dt/2 L(u); u2 = u1 + dt/2 L(u1); u3 = 2/3 u + 1/3 u2 + dt/6 L(u2); u4 = u3 + dt/2 L(u3)
    const Stage s12{0.0, 1.0, 0.5, 0};
    const Stage s3{2.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0, 0};
    for (int s = 0; s < nsteps; ++s) {
        if (s == 1 && nsteps > 2 && steady_step_graph(e, mode, cfl_h)) {
            for (; s < nsteps; ++s) {
                HYPE_CK(cudaGraphLaunch(e->step_graph, e->stream));
                count_launch(e->graph_launches);
            }
            break;
        }
        if (s == 0 && first_from_rhs) {
            // the initial RHS call of hype.c:175 is this step's first stage RHS
            if ((rc = launch_first_stage_from_rhs(e, mode, cfl_h, s12))) return rc;
        } else {
            // dt: MONITOR refreshes it from the last stage of the previous step
            const int use_src = (mode == HYPE_DT_MONITOR) && s > 0;
            k_begin_step<<<1, 1, 0, e->stream>>>(e->ds, mode, 3, use_src, 1, cfl_h, e->p.recon, 1.0 / e->p.h,
                                                 e->C4 != nullptr);
            HYPE_LAUNCHED(1);
            if ((rc = launch_stage(e, e->U, e->U, e->U, e->W, s12, 0))) return rc;
        }
        if ((rc = launch_stage(e, e->W, e->U, e->W, e->W, s12, 1))) return rc;
        if ((rc = launch_stage(e, e->W, e->U, e->W, e->W, s3, 2))) return rc;
        if ((rc = launch_stage(e, e->W, e->U, e->W, e->U, s12, 3))) return rc;
    }
    if ((rc = read_scalars(e))) return rc;
    *t_inout = e->hs->t;
    const double smax3 = bits_to_double(e->hs->smax_bits[3]);
    if (nsteps > 0 && mode == HYPE_DT_MONITOR)
        *dt_inout = cfl_dt(cfl_h, smax3, e->p.recon, bits_to_double(e->hs->smaxv_bits[3]), 1.0 / e->p.h,
                           e->C4 != nullptr);
    else
        *dt_inout = e->hs->dt;
    if (st) {
        st->bad_cell = e->hs->bad == ~0ull ? -1 : (long long)e->hs->bad;
        st->smax = smax3;
        st->rhs_evals = 4LL * nsteps;
    }
    return e->hs->bad == ~0ull ? HYPE_OK : HYPE_ERR_STATE;
}

extern "C" void* hype_euler_stream(hype_euler* e) { return e ? (void*)e->stream : nullptr; }

extern "C" int hype_euler_monitor(hype_euler* e, double* ke, double* dissipation) {
    if (!e || !ke || !dissipation) return HYPE_ERR_ARG;
    constexpr int kMaxBlocks = 152 * 8;
    const int nblk = (int)std::min<long long>(kMaxBlocks, (e->g.N + kMonThreads - 1) / kMonThreads);
    if (!e->mon) HYPE_CK(cudaMalloc((void**)&e->mon, sizeof(double) * (2 * kMaxBlocks + 2)));
    const double h = e->p.h;
    k_monitor<<<nblk, kMonThreads, 0, e->stream>>>(e->U, e->g, h * h * h, 0.5 / h, e->p.mu, e->mon);
    k_monitor_sum<<<1, kMonThreads, 0, e->stream>>>(e->mon, nblk, e->mon + 2 * kMaxBlocks);
    HYPE_LAUNCHED(2);
    double r[2];
    HYPE_CK(cudaMemcpyAsync(r, e->mon + 2 * kMaxBlocks, sizeof(r), cudaMemcpyDeviceToHost, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    *ke = r[0];
    *dissipation = r[1];
    return HYPE_OK;
}

extern "C" int hype_euler_set_mlp(hype_euler* e, const float* params, float prob_threshold) {
    if (!e || !params || !(prob_threshold > 0.0f) || !(prob_threshold < 1.0f)) return HYPE_ERR_ARG;
    std::vector<__nv_bfloat16> h(mlp::NPARAM);
    for (int q = 0; q < mlp::NPARAM; ++q) h[q] = __float2bfloat16_rn(params[q]);
    mlp::MmaWeights hw;  // host staging, copied before the stream synchronisation below
    mlp::pack_weights(h.data(), hw);
    // before the network, whose presence lets the gated kernels run
    if (!e->bound64 && e->p.precision != HYPE_PREC_FP32) {
        if (!e->flag64) HYPE_CK(cudaMalloc((void**)&e->flag64, (size_t)e->g.NE));
        // the bounds lie in the staging array of the host copies, which are in the same stream; grids under 8 cells
        // a side need one of their own
        const size_t need = sizeof(float) * NV * (size_t)e->g.NE;
        if (need <= sizeof(double) * NV * (size_t)e->g.N) e->bound64 = (float*)e->stage_aos;
        else HYPE_CK(cudaMalloc((void**)&e->bound64, need));
    }
    if (!e->mlp) HYPE_CK(cudaMalloc((void**)&e->mlp, sizeof(mlp::MmaWeights)));
    if (!e->gate && e->p.precision == HYPE_PREC_FP32) {
        HYPE_CK(cudaMalloc((void**)&e->gate, (size_t)e->g.NE));
        HYPE_CK(cudaMalloc((void**)&e->gate_wide, (size_t)e->g.NE));
        HYPE_CK(cudaMemsetAsync(e->gate, 0, (size_t)e->g.NE, e->stream));
        HYPE_CK(cudaMemsetAsync(e->gate_wide, 0, (size_t)e->g.NE, e->stream));
    }
    HYPE_CK(cudaMemcpyAsync(e->mlp, &hw, sizeof(mlp::MmaWeights), cudaMemcpyHostToDevice, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    e->logit_thr = logf(prob_threshold / (1.0f - prob_threshold));
    return HYPE_OK;
}

extern "C" int hype_euler_set_gate_per_step(hype_euler* e, int per_step) {
    if (!e || (per_step != 0 && per_step != 1)) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    e->gate_per_step = per_step;  // part of the step graph's key: the next step recaptures
    return HYPE_OK;
}

extern "C" int hype_euler_gate_flags(hype_euler* e, unsigned char* out, int widened) {
    if (!e || !out || (widened != 0 && widened != 1)) return HYPE_ERR_ARG;
    if (!e->gate) return HYPE_ERR_UNSUPPORTED;
    HYPE_CK(cudaMemcpyAsync(out, widened ? e->gate_wide : e->gate, (size_t)e->g.NE, cudaMemcpyDeviceToHost, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    return HYPE_OK;
}

extern "C" int hype_euler_indicator_stats(hype_euler* e, long long* flagged, long long* positivity_fallbacks, int reset) {
    if (!e) return HYPE_ERR_ARG;
    unsigned long long c[2];
    HYPE_CK(cudaMemcpyAsync(c, e->mlp_cnt, sizeof(c), cudaMemcpyDeviceToHost, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    if (flagged) *flagged = (long long)c[0];
    if (positivity_fallbacks) *positivity_fallbacks = (long long)c[1];
    if (reset) HYPE_CK(cudaMemsetAsync(e->mlp_cnt, 0, sizeof(c), e->stream));
    return HYPE_OK;
}

extern "C" int hype_euler_set_recon(hype_euler* e, int recon) {
    if (!e || recon < HYPE_RECON_CWENO4 || recon > HYPE_RECON_WENO3) return HYPE_ERR_ARG;
    if (e->C4 && recon == HYPE_RECON_LEARNED) return HYPE_ERR_ARG;  // the viscous path keeps the R4 coefficients
    if (e->p.precision == HYPE_PREC_DF64 && recon == HYPE_RECON_WENO3) return HYPE_ERR_UNSUPPORTED;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    e->p.recon = recon;
    return HYPE_OK;
}

extern "C" int hype_euler_sample_features(hype_euler* e, long long stride, float* X, float* D, long long* ns_out) {
    if (!e || stride < 1 || !X || !D) return HYPE_ERR_ARG;
    const long long ns = (e->g.N + stride - 1) / stride;
    float *dX = nullptr, *dD = nullptr;
    cudaError_t ce = cudaMalloc((void**)&dX, sizeof(float) * ns * 3 * mlp::NIN);
    if (ce == cudaSuccess) ce = cudaMalloc((void**)&dD, sizeof(float) * ns);
    if (ce == cudaSuccess) {
        k_features<<<cdiv(ns, 128), 128, 0, e->stream>>>(e->U, e->g, stride, ns, dX, dD);
        count_launch(1);
        ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(X, dX, sizeof(float) * ns * 3 * mlp::NIN, cudaMemcpyDeviceToHost, e->stream);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(D, dD, sizeof(float) * ns, cudaMemcpyDeviceToHost, e->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(e->stream);
    cudaFree(dX);
    cudaFree(dD);
    if (ce != cudaSuccess) {
        set_last_error("hype_euler_sample_features", ce);
        return HYPE_ERR_CUDA;
    }
    if (ns_out) *ns_out = ns;
    return HYPE_OK;
}

extern "C" int hype_euler_set_stage_kernel(hype_euler* e, int mode) {
    if (!e || (mode != HYPE_STAGE_AUTO && mode != HYPE_STAGE_UNFUSED)) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    e->stage_mode = mode;
    return prepare(e);
}

extern "C" int hype_euler_profile(hype_euler* e, int enable) {
    if (!e) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    e->prof = enable != 0;
    e->ev_used = 0;
    return HYPE_OK;
}

extern "C" int hype_euler_profile_read(hype_euler* e, double* ms, long long* count) {
    if (!e || !ms || !count) return HYPE_ERR_ARG;
    HYPE_CK(cudaStreamSynchronize(e->stream));
    for (int k = 0; k < 3; ++k) {
        ms[k] = 0.0;
        count[k] = 0;
    }
    for (size_t q = 0; q + 1 < e->ev_used + 1 && q < e->ev_used; q += 2) {
        float t = 0.0f;
        HYPE_CK(cudaEventElapsedTime(&t, e->ev[q], e->ev[q + 1]));
        ms[e->ev_kind[q / 2]] += t;
        count[e->ev_kind[q / 2]] += 1;
    }
    return HYPE_OK;
}

// ======================================================================
// Allocation-free RHS evaluation.
//
// Some callers cannot let a plugin allocate device memory: hosts that hand the
// plugin pre-allocated device vectors and own every byte of device memory
// through their own pool, and latency-critical loops where cudaMalloc's
// implicit device-wide synchronisation is not acceptable.  For them,
// hype_euler_rhs_noalloc runs the same three kernels as hype_euler_rhs_device
// with all of their scratch (face traces, face fluxes, the wave-speed and
// admissibility words) in the fixed device array below, which every GPU that
// loads this library holds until the process exits.
namespace hype {
namespace euler {

constexpr long long kNoAllocMaxExt = 18LL * 18 * 18;  // (nx+2)(ny+2)(nz+2) <= 5832, e.g. 16^3 cells
constexpr size_t kAlign = 256;
constexpr size_t align_up(size_t b) { return (b + kAlign - 1) / kAlign * kAlign; }
constexpr size_t kNoAllocTraceBytes = align_up(sizeof(double) * NV * NTR * kNoAllocMaxExt);
constexpr size_t kNoAllocFluxBytes = align_up(sizeof(double) * NV * kNoAllocMaxExt);  // one direction
constexpr size_t kNoAllocScalarBytes = align_up(sizeof(DevScalars));
// the reconstruction's two event counters (indicator, positivity fallback): written, never read here
constexpr size_t kNoAllocCounterBytes = align_up(2 * sizeof(unsigned long long));
// ghosted stage input: (nx+6)(ny+6)(nz+6) <= (9/5)^3 (nx+2)(ny+2)(nz+2) for n >= 3
constexpr long long kNoAllocMaxGhost = kNoAllocMaxExt * 729 / 125 + 1;
constexpr size_t kNoAllocGhostBytes = align_up(sizeof(double) * NV * kNoAllocMaxGhost);
constexpr size_t kNoAllocBytes = kNoAllocTraceBytes + 3 * kNoAllocFluxBytes + kNoAllocScalarBytes +
                                 kNoAllocCounterBytes + kNoAllocGhostBytes;  // ~7.7 MB

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

}  // namespace euler
}  // namespace hype

#include <mutex>

static std::mutex g_noalloc_mutex;
static void* g_noalloc_base[128] = {nullptr};

extern "C" long long hype_euler_noalloc_max_ext(void) { return kNoAllocMaxExt; }

extern "C" int hype_euler_rhs_noalloc(const hype_euler_params* p, const double* dU, double* dRHS, double* dt_out,
                                      void* stream) {
    if (!p || !dU || !dRHS) return HYPE_ERR_ARG;
    if (p->nx < 3 || p->ny < 3 || p->nz < 3 || !(p->h > 0) || !(p->cfl > 0) || !(p->gamma > 1.0)) return HYPE_ERR_ARG;
    for (int f = 0; f < 6; ++f)
        if (p->bc[f] < HYPE_BC_PERIODIC || p->bc[f] > HYPE_BC_TRANSMISSIVE) return HYPE_ERR_ARG;
    for (int d = 0; d < 3; ++d)
        if ((p->bc[2 * d] == HYPE_BC_PERIODIC) != (p->bc[2 * d + 1] == HYPE_BC_PERIODIC)) return HYPE_ERR_ARG;
    if (p->recon != HYPE_RECON_CWENO4 && p->recon != HYPE_RECON_LINEAR4 && p->recon != HYPE_RECON_WENO3) return HYPE_ERR_ARG;
    if (p->precision != HYPE_PREC_FP64 && p->precision != HYPE_PREC_FP32) return HYPE_ERR_ARG;
    if (p->flux < HYPE_FLUX_RUSANOV || p->flux > HYPE_FLUX_ROTHLLC) return HYPE_ERR_ARG;
    if (p->positivity != 0 && p->positivity != 1) return HYPE_ERR_ARG;
    if (p->mu != 0.0) {
        set_last_error("hype_euler_rhs_noalloc: the viscous terms need a context (hype_euler_create)", cudaErrorInvalidValue);
        return HYPE_ERR_UNSUPPORTED;
    }
    const long long ne = (long long)(p->nx + 2) * (p->ny + 2) * (p->nz + 2);
    if (ne > kNoAllocMaxExt) {
        set_last_error("hype_euler_rhs_noalloc: grid exceeds the fixed scratch ((nx+2)(ny+2)(nz+2) > 5832)",
                       cudaErrorInvalidValue);
        return HYPE_ERR_ARG;
    }
    // one-time set-up per device, with that device current: the device address of the
    // scratch array (its name is only a host-side stand-in in host code)
    int dev = 0;
    HYPE_CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) return HYPE_ERR_UNSUPPORTED;
    unsigned char* base;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mutex);
        if (!g_noalloc_base[dev]) {
            void* ptr = nullptr;
            cudaError_t ce = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
            if (ce != cudaSuccess) {
                set_last_error("cudaGetSymbolAddress", ce);
                return HYPE_ERR_CUDA;
            }
            g_noalloc_base[dev] = ptr;
        }
        base = (unsigned char*)g_noalloc_base[dev];
    }
    Geo g;
    g.nx = p->nx; g.ny = p->ny; g.nz = p->nz;
    for (int f = 0; f < 6; ++f) g.bc[f] = p->bc[f];
    g.N = (long long)p->nx * p->ny * p->nz;
    g.NE = ne;
    g.ex = p->nx + 2;
    g.ey = p->ny + 2;
    set_ghost_extents(g);
    void* T = base;
    double* Fx = (double*)(base + kNoAllocTraceBytes);
    double* Fy = (double*)(base + kNoAllocTraceBytes + kNoAllocFluxBytes);
    double* Fz = (double*)(base + kNoAllocTraceBytes + 2 * kNoAllocFluxBytes);
    DevScalars* ds = (DevScalars*)(base + kNoAllocTraceBytes + 3 * kNoAllocFluxBytes);
    unsigned long long* counters =
        (unsigned long long*)(base + kNoAllocTraceBytes + 3 * kNoAllocFluxBytes + kNoAllocScalarBytes);
    void* G = base + kNoAllocTraceBytes + 3 * kNoAllocFluxBytes + kNoAllocScalarBytes + kNoAllocCounterBytes;
    cudaStream_t s = (cudaStream_t)stream;
    // the scratch keeps the previous call's contents: the wave-speed maximum and the
    // admissibility word must start cleared; traces and fluxes are fully rewritten
    k_reset_slot<<<1, 1, 0, s>>>(ds, 4);
    HYPE_CK(cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), s));
    const dim3 br(32, 4), gr(cdiv(g.nx + 2, 32), cdiv(g.ny + 2, 4), g.nz + 2);
    const int rec = p->recon;
    const int pad = p->positivity;
    if (p->precision == HYPE_PREC_FP32) {
        // the FP32 admissibility check of the positivity fallback keeps its per-warp columns in
        // dynamic shared memory, as in the context path
        const size_t ck_bytes = pad ? sizeof(float) * 4 * 2 * NTR * 32 : 0;
        k_ghost<float><<<ghost_grid(g), kGhostThreads, 0, s>>>(dU, (float*)G, g);
        k_recon_f32<<<gr, br, ck_bytes, s>>>((const float*)G, (float*)T, g, rec, pad, p->gamma - 1.0, counters);
    } else {
        k_ghost<double><<<ghost_grid(g), kGhostThreads, 0, s>>>(dU, (double*)G, g);
        launch_recon64(g, (const double*)G, (double*)T, rec, pad, p->gamma - 1.0, counters, nullptr, s);
    }
    const int nfk = launch_faces(g, T, Fx, Fy, Fz, p->gamma, ds, 4, p->precision == HYPE_PREC_FP32, p->flux, s);
    const Stage st{0.0, 0.0, 0.0, 1};
    const unsigned bu = kUpdateThreads;
    const dim3 gu = update_grid(g);
    if (p->precision == HYPE_PREC_FP32)
        k_update<true><<<gu, bu, 0, s>>>(Fx, Fy, Fz, nullptr, nullptr, dRHS, g, 1.0 / p->h, st, ds);
    else
        k_update<false><<<gu, bu, 0, s>>>(Fx, Fy, Fz, nullptr, nullptr, dRHS, g, 1.0 / p->h, st, ds);
    HYPE_LAUNCHED(4 + nfk);
    if (dt_out) {
        unsigned long long w[2];
        HYPE_CK(cudaMemcpyAsync(&w[0], &ds->smax_bits[4], sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        HYPE_CK(cudaMemcpyAsync(&w[1], &ds->bad, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        HYPE_CK(cudaStreamSynchronize(s));
        *dt_out = cfl_dt(p->cfl * p->h, bits_to_double(w[0]), p->recon);
        if (w[1] != ~0ull) return HYPE_ERR_STATE;
    }
    return HYPE_OK;
}

// One step of the current reconstruction and, from the same state, one full-CWENO4
// step; keeps the first, returns the relative L1 difference of the densities.
extern "C" int hype_euler_shadow_step(hype_euler* e, double* t_inout, double* dt_inout, double* l1_rel) {
    if (!e || !t_inout || !dt_inout || !l1_rel) return HYPE_ERR_ARG;
    const size_t bytes = sizeof(double) * NV * (size_t)e->g.N;
    const int recon = e->p.recon;
    const double t0 = *t_inout, dt0 = *dt_inout;
    HYPE_CK(cudaMemcpyAsync(e->S, e->U, bytes, cudaMemcpyDeviceToDevice, e->stream));
    e->p.recon = HYPE_RECON_CWENO4;
    double t = t0, dt = dt0;
    int rc = hype_euler_step(e, 1, &t, &dt, nullptr);
    e->p.recon = recon;
    if (rc) return rc;
    HYPE_CK(cudaMemcpyAsync(e->L, e->U, sizeof(double) * (size_t)e->g.N, cudaMemcpyDeviceToDevice, e->stream));
    HYPE_CK(cudaMemcpyAsync(e->U, e->S, bytes, cudaMemcpyDeviceToDevice, e->stream));
    *t_inout = t0;
    *dt_inout = dt0;
    if ((rc = hype_euler_step(e, 1, t_inout, dt_inout, nullptr))) return rc;
    double* acc = e->acc;
    HYPE_CK(cudaMemsetAsync(acc, 0, 2 * sizeof(double), e->stream));
    k_l1<<<608, 256, 0, e->stream>>>(e->U, e->L, e->g.N, acc);
    HYPE_LAUNCHED(1);
    double h[2];
    HYPE_CK(cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, e->stream));
    HYPE_CK(cudaStreamSynchronize(e->stream));
    *l1_rel = h[0] / h[1];
    return HYPE_OK;
}
