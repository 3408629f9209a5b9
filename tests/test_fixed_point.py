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
