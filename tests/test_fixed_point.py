"""The integer arithmetic of the FP64 kernels (csrc/fixed.cuh, the face states of csrc/cweno_fix.cuh), whose functions
are host functions too, against exact rational arithmetic."""
import ctypes as C
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from acoustic_petsc_gb300 import _build
from conftest import ROOT


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed") / "fixed_host.so")
    subprocess.run([_build.nvcc(), *_build.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "-I", _build.CSRC, os.path.join(ROOT, "tests", "fixed_host.cu"), "-o", so], check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _call(host, name, a, b=None):
    a = np.ascontiguousarray(a)
    b = a if b is None else np.ascontiguousarray(b)
    out = np.empty_like(a)
    getattr(host, name)(C.c_int(a.size), _p(a), _p(b), _p(out))
    return out


def _numbers(rng, n, lo, hi):
    """significands at random, all ones, one, and one bit, with exponents over [lo, hi)"""
    m = 1.0 + rng.random(n)
    m[: n // 8] = np.nextafter(2.0, 0.0)
    m[n // 8: n // 4] = 1.0
    m[n // 4: n // 2] = 1.0 + 2.0 ** -rng.integers(1, 53, n // 2 - n // 4)
    return np.ldexp(m, rng.integers(lo, hi, n))


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, -1e-310, 1.7976931348623157e308, 1.0, -3.0])


def test_division_and_root_are_ieee_ones(host):
    """div_rn and sqrt_rn round as the IEEE operations do, every class of operand included"""
    rng = np.random.default_rng(1)
    a = np.concatenate([_numbers(rng, 20000, -1074, 1024), -_numbers(rng, 20000, -300, 300), np.repeat(SPECIAL, SPECIAL.size)])
    b = np.concatenate([_numbers(rng, 20000, -1074, 1024), _numbers(rng, 20000, -300, 300), np.tile(SPECIAL, SPECIAL.size)])
    p = rng.permutation(40000)
    a[:40000] = a[:40000][p]
    with np.errstate(all="ignore"):
        want, root = a / b, np.sqrt(a)
    for got, ref in ((_call(host, "t_div_rn", a, b), want), (_call(host, "t_sqrt_rn", a), root)):
        same = (got.view(np.uint64) == ref.view(np.uint64)) | (np.isnan(got) & np.isnan(ref))
        assert same.all(), (a[~same][:4], b[~same][:4])


def test_reciprocal_and_roots(host):
    """within 0.52 of a unit in the last place: the rounding's half and the 2^-59 before it (2^-6 of a unit)"""
    rng = np.random.default_rng(2)
    x = _numbers(rng, 4000, -1000, 1000)
    for v, y in zip(x, _call(host, "t_recip", x)):
        assert abs(1 / Fraction(v) - Fraction(y)) <= Fraction(0.52) * Fraction(math.ulp(y))
    half = Fraction(0.52)
    for v, y, r in zip(x, _call(host, "t_sqrt", x), _call(host, "t_rsqrt", x)):
        u, w = half * Fraction(math.ulp(y)), half * Fraction(math.ulp(r))
        assert (Fraction(y) - u) ** 2 <= Fraction(v) <= (Fraction(y) + u) ** 2
        assert (Fraction(r) - w) ** 2 <= 1 / Fraction(v) <= (Fraction(r) + w) ** 2


def _sides(host, q, gamma):
    q = np.ascontiguousarray(q)
    out = np.empty((len(q), 4))
    host.t_side(C.c_int(len(q)), _p(q), C.c_double(gamma), _p(out))
    return out


def test_face_states(host):
    """velocity, pressure and |u| + c of a face state where side_fix takes it.  Each is formed to 2^-59 of its largest
    part, then rounded: 2^-52 of u and of |u| + c, and for p of (gamma - 1) (E + |m|^2 / 2 rho)"""
    rng = np.random.default_rng(3)
    n = 3000
    rho = _numbers(rng, n, -44, 199)
    m = rng.choice([-1.0, 1.0], (n, 3)) * np.ldexp(1.0 + rng.random((n, 3)), rng.integers(-60, 3, (n, 3)))
    m *= rho[:, None]
    m[:200] = 0.0
    E = 0.5 * (m ** 2).sum(-1) / rho + rho * np.ldexp(1.0 + rng.random(n), rng.integers(-8, 8, n))
    out = _sides(host, np.column_stack([rho, m, E]), 1.4)
    assert out[:, 0].sum() >= 0.5 * n
    g, g1 = Fraction(1.4), Fraction(1.4 - 1.0)
    for k in range(n):
        if not out[k, 0]:
            continue
        r, e, mm = Fraction(rho[k]), Fraction(E[k]), [Fraction(v) for v in m[k]]
        un, kin = mm[0] / r, sum(v * v for v in mm) / (2 * r)
        p = g1 * (e - kin)
        assert abs(Fraction(out[k, 1]) - un) <= abs(un) * Fraction(2) ** -52
        assert abs(Fraction(out[k, 2]) - p) <= g1 * (e + kin) * Fraction(2) ** -52
        c = Fraction(out[k, 3]) - abs(un)  # c^2 = gamma p / rho, to the error that p may have
        tol = Fraction(out[k, 3]) * Fraction(2) ** -52
        slack = g * g1 * (e + kin) / r * Fraction(2) ** -56
        assert (c - tol) ** 2 <= g * p / r + slack and (c + tol) ** 2 >= g * p / r - slack


@pytest.mark.parametrize("rho", [8.0, 1e3, 1e6, 2.0 ** 199, 0.7, 1.5])
def test_face_states_of_vanishing_momenta(host, rho):
    """velocities down to the smallest numbers: m / rho to 2^-52, or, where it or the momentum is not a normal number,
    zero with the momentum's sign"""
    mn = np.concatenate([10.0 ** np.arange(-300.0, -307.5, -0.25), [5e-308, 3e-308, 2.3e-308, 2.2250738585072014e-308,
                                                                      1e-308, 1e-310, 5e-324, 0.0]])
    mn = np.concatenate([mn, -mn])
    q = np.zeros((mn.size, 5))
    q[:, 0], q[:, 1], q[:, 4] = rho, mn, 2.5 * rho
    out = _sides(host, q, 1.4)
    want = mn / rho
    assert out[:, 0].all() and (np.signbit(out[:, 1]) == np.signbit(mn)).all()
    normal = (np.abs(want) >= 2.0 ** -1020) & (np.abs(mn) >= 2.0 ** -1022)
    assert (np.abs(out[normal, 1] - want[normal]) <= 2.0 ** -52 * np.abs(want[normal])).all()
    assert (np.abs(out[~normal, 1]) <= np.abs(want[~normal]) * (1 + 2.0 ** -52)).all()
    assert (np.abs(out[:, 2] - 0.4 * 2.5 * rho) <= 1e-15 * rho).all()


def _exact_traces(s, at, linear):
    """the 24 face traces of the CWENO4 (or R4) polynomial of n stencils in extended precision, as weno() and
    evaluate_polynomial define them (3d/weno4/Viscous-Multiphase-Fourth-Order/reconstruction.c:12-259); at: the
    offsets of the 33 values"""
    LD = np.longdouble
    u = {tuple(at[i]): s[:, i].astype(LD) for i in range(33)}

    def v(**k):
        return u[tuple(k.get(c, 0) for c in "xyz")]

    ax, pairs = "xyz", [("x", "y"), ("y", "z"), ("z", "x")]
    u0 = v()
    d4 = [(11 * v(**{a: -2}) - 82 * v(**{a: -1}) + 82 * v(**{a: 1}) - 11 * v(**{a: 2})) / LD(120) for a in ax]
    dd = [(v(**{a: -1}) - 2 * u0 + v(**{a: 1})) / 2 for a in ax]
    d3 = [(-v(**{a: -2}) + 2 * (v(**{a: -1}) - v(**{a: 1})) + v(**{a: 2})) / LD(12) for a in ax]
    d1 = [(v(**{a: 1}) - v(**{a: -1})) / 2 for a in ax]

    def x(a, b, first):  # the difference along b of the values one cell towards `first` of a
        return v(**{a: first, b: 1}) - v(**{a: first, b: -1})

    cross = [(x(a, b, 1) - x(a, b, -1)) / 4 for a, b in pairs]
    aab = {(a, b): (x(a, b, 1) + x(a, b, -1)) / 4 - d1[ax.index(b)] for a in ax for b in ax if a != b}
    xyz = sum(p * q * r * v(x=p, y=q, z=r) for p in (-1, 1) for q in (-1, 1) for r in (-1, 1)) / LD(8)
    one = [(d1, dd, cross)]
    for i, a in enumerate(ax):
        for sg in (1, -1):
            d, e, c = list(d1), list(dd), list(cross)
            d[i] = sg * (-3 * u0 + 4 * v(**{a: sg}) - v(**{a: 2 * sg})) / LD(2)
            e[i] = (u0 - 2 * v(**{a: sg}) + v(**{a: 2 * sg})) / 2
            for j, b in enumerate(ax):
                if b != a:
                    k = next(n for n, p in enumerate(pairs) if set(p) == {a, b})
                    c[k] = sg * (x(a, b, sg) / 2 - d1[j])
            one.append((d, e, c))
    sq = lambda t: sum(q * q for q in t)  # noqa: E731
    wr, l0, e0, c0 = LD(1), d4, dd, cross
    if not linear:
        is4 = sq(d4) + LD(13) / 3 * sq(dd) + LD(7) / 6 * sq(cross) + sum(p * q for p, q in zip(d4, d3)) / LD(5) + LD(47) / 10 * sq(aab.values()) + \
            LD(3906) / 100 * sq(d3) + LD(61) / 48 * xyz * xyz
        g, eps = LD(85) / 100, LD(1) / 10 ** 12
        gk = [(1 - g) * g] + 6 * [(1 - g) ** 2 / 6]
        w = [gk[k] / (sq(d) + LD(13) / 3 * sq(e) + LD(7) / 6 * sq(c) + eps) ** 4 for k, (d, e, c) in enumerate(one)]
        w4 = g / (is4 + eps) ** 4
        tot = w4 + sum(w)
        w, wr = [q / tot for q in w], w4 / tot / g
        mix = lambda n, i, r4: sum((w[k] - wr * gk[k]) * one[k][n][i] for k in range(7)) + wr * r4[i]  # noqa: E731
        l0, e0, c0 = ([mix(n, i, r4) for i in range(3)] for n, r4 in enumerate((d4, dd, cross)))
    r12, r320 = LD(1) / 12, LD(3) / 20
    gp = np.sqrt(LD(3)) / 6
    out = np.empty((len(s), 24), dtype=LD)
    for q in range(24):
        D, hi, s1, s2 = q >> 3, (q >> 2) & 1, (q >> 1) & 1, q & 1
        X = [None] * 3
        X[D] = LD(hi) - LD(1) / 2
        t = [a for a in range(3) if a != D]
        X[t[0]], X[t[1]] = (gp if s1 else -gp), (gp if s2 else -gp)
        y = u0 + sum(l0[a] * X[a] + e0[a] * (X[a] ** 2 - r12) + wr * d3[a] * X[a] * (X[a] ** 2 - r320) for a in range(3))
        y = y + sum(c * X[ax.index(a)] * X[ax.index(b)] for c, (a, b) in zip(c0, pairs)) + wr * xyz * X[0] * X[1] * X[2]
        for (a, b), c in aab.items():
            y = y + wr * c * (X[ax.index(a)] ** 2 - r12) * X[ax.index(b)]
        out[:, q] = y
    return out


@pytest.fixture(scope="module")
def offsets(host):
    at = (C.c_int * 99)()
    host.t_stencil(at)
    return np.array(at).reshape(33, 3)


@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("strict", [0, 1])
@pytest.mark.parametrize("quiet", [1.0, 0.3, 0.1, 1 / 17, 1e-2, 1e-3, 1e-6, 1e-12, 0.0])
def test_reconstruction_of_a_quiet_cell_beside_a_jump(host, offsets, linear, strict, quiet):
    """the traces where the fixed-point form takes the stencil, against extended precision.  The values' units are
    2^-58 of the largest one's power of two and the smoothness indicators' 2^-55, which moves weights between the
    stencils by 2^-52 or so of it (2.2e-16): 4e-16 of the largest.  A polynomial that the weights leave below 2^-6 of
    the largest, and with `strict` (density, energy, pressure) a cell four binary exponents below it, is left to the
    FP64 form, and R4 keeps 1/64 of the largest in its traces: 64 (`strict`: 16) times as much of the traces or the
    cell, however small they are"""
    rng = np.random.default_rng(7)
    n = 1500
    normal = rng.standard_normal((n, 3))
    normal[: n // 3] = np.eye(3)[rng.integers(0, 3, n // 3)]
    normal /= np.linalg.norm(normal, axis=1)[:, None]
    beyond = (normal @ offsets.T) > rng.uniform(0.05, 1.9, (n, 1))
    s = np.where(beyond, 1.0, quiet) * (1 + rng.choice([1e-3, 0.3], (n, 1)) * rng.uniform(-1, 1, (n, 33)))
    s = np.ascontiguousarray(s[beyond.any(axis=1)])
    out = np.zeros((len(s), 25))
    host.t_recon(C.c_int(len(s)), _p(s), C.c_int(linear), C.c_int(strict), _p(out))
    taken = out[:, 0] != 0
    assert quiet < 0.1 or taken.all() or strict
    assert not taken.any() if strict and quiet <= 1e-2 else True
    err = np.abs(out[:, 1:] - _exact_traces(s, offsets, linear)).max(axis=1)[taken]
    size = np.maximum(np.abs(out[:, 1:]).max(axis=1), np.abs(s[:, 0]))[taken]
    assert (err <= 4e-16 * np.abs(s).max(axis=1)[taken]).all()
    assert (err <= 4e-16 * (16 if strict else 64) * size).all()
    if taken.any():
        print(f"linear {linear} strict {strict} quiet {quiet:g}: {taken.mean():.3f} taken, {float((err / size).max()):.2e} of the traces")


@pytest.mark.parametrize("linear", [0, 1])
def test_reconstruction_of_small_stencils(host, offsets, linear):
    """a stencil of zeros gives zeros; one whose every value is below 2^-959 is held in units of 2^-1017 (a few of them
    off in the traces), one that is not finite is left to the FP64 form; and smooth stencils through zero are taken"""
    rng = np.random.default_rng(8)
    s = np.zeros((6, 33))
    s[1] = 1e-300 * rng.uniform(0.5, 1, 33)
    s[2] = np.nan
    s[3, 7] = np.inf
    s[4] = offsets @ [0.3, -0.2, 0.1]
    s[5] = np.sin(offsets @ [0.3, -0.2, 0.1] + 0.01)
    out = np.zeros((6, 25))
    host.t_recon(C.c_int(6), _p(s), C.c_int(linear), C.c_int(0), _p(out))
    assert list(out[:, 0]) == [1, 1, 0, 0, 1, 1] and not out[0, 1:].any()
    # the differences are far below 1e-12, so the weights are R4's
    assert np.abs(out[1:2, 1:] - _exact_traces(s[1:2], offsets, 1)).max() <= 2.0 ** -1013
    assert np.abs(out[4:, 1:] - _exact_traces(s[4:], offsets, linear)).max() <= 4e-16
