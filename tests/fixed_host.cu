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
