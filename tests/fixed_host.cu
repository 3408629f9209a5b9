// Host builds of the integer arithmetic (fixed.cuh, cweno_fix.cuh) for test_fixed_point.py.
#include "cweno_fix.cuh"

using namespace hype::euler;

#define EACH(name, expr)                                                                        \
    extern "C" void name(int n, const double* a, const double* b, double* out) {                \
        for (int i = 0; i < n; ++i) out[i] = expr;                                              \
        (void)b;                                                                                \
    }
EACH(t_recip, recip_fix(a[i]))
EACH(t_sqrt, sqrt_fix(a[i]))
EACH(t_rsqrt, rsqrt_fix(a[i]))
EACH(t_div_rn, div_rn(a[i], b[i]))
EACH(t_sqrt_rn, sqrt_rn(a[i]))

// q: n rows (rho, normal momentum, two tangential ones, E); out: n rows (taken, un, p, |un| + c)
extern "C" void t_side(int n, const double* q, double gamma, double* out) {
    for (int i = 0; i < n; ++i) {
        const double* s = q + 5 * i;
        double* o = out + 4 * i;
        o[1] = o[2] = o[3] = 0.0;
        o[0] = side_fix(s[0], s[1], s[2], s[3], s[4], gamma, gamma - 1.0, o[1], o[2], o[3]);
    }
}

// n stencils of 33 values (the order of S1, SQ, SO); out: n rows of whether the fixed-point form takes it and its 24 traces
template <bool LINEAR>
static void recon(int n, const double* s, int strict, double* out) {
    PolyFix p;
    for (int i = 0; i < n; ++i) out[25 * i] = recon_fix<LINEAR>(s + 33 * i, strict != 0, out + 25 * i + 1, 1, p);
}
extern "C" void t_recon(int n, const double* s, int linear, int strict, double* out) {
    linear ? recon<true>(n, s, strict, out) : recon<false>(n, s, strict, out);
}
// the offset of each of the 33 values
extern "C" void t_stencil(int* at) {
    for (int i = 0; i < 99; ++i) at[i] = 0;
    for (int a = 0; a < 3; ++a)
        for (int o = -2; o <= 2; ++o)
            if (o) at[3 * S1(a, o) + a] = o;
    for (int a = 0; a < 3; ++a)
        for (int b = a + 1; b < 3; ++b)
            for (int q = 0; q < 4; ++q) {
                int* c = at + 3 * SQ(a, q >> 1, b, q & 1);
                c[a] = 2 * (q >> 1) - 1;
                c[b] = 2 * (q & 1) - 1;
            }
    for (int q = 0; q < 8; ++q)
        for (int a = 0; a < 3; ++a) at[3 * SO(q >> 2, (q >> 1) & 1, q & 1) + a] = 2 * ((q >> (2 - a)) & 1) - 1;
}
