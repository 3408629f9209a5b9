"""Performance cases: the calls that programs on this framework make, timed as they make them.

A case is one solver at one size with its options.  ``prepare`` builds what such a program holds (the solver
handle with the initial state resident on the GPU), ``run`` makes one pass (a few time steps and the state
they leave, or one right-hand side), ``work`` counts what the pass cannot do without, and ``exact`` gives the
same result from plain 64-bit tensor operations, without the framework's kernels.

A pass continues from the state that the last one left, as a time loop does; after ``horizon`` steps the run
is over and the next pass starts again from the initial state.
"""
import math

import numpy as np
import torch

import acoustic_petsc_gb300 as H
from acoustic_petsc_gb300 import _lib as L

FP64, FP32, DF64 = L.PREC_FP64, L.PREC_FP32, L.PREC_DF64
PER, REF, TRA, ZERO, ADI = L.BC_PERIODIC, L.BC_REFLECTIVE, L.BC_TRANSMISSIVE, L.BC_ZERO, L.BC_ADIABATIC
WATER_AIR = (4.4, 6.0e8, 1.4, 0.0)
TWO_GASES = (1.4, 0.0, 1.6, 0.0)
GP = 0.28867513459481287


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest grid of the test and start-up runs: launches and latency count
        dict(name="euler_16_fp64", kind="euler", nx=16, ny=16, nz=16, prec="fp64", init="pulse", bc="periodic", steps=8),
        # RHSFunction as a PETSc host program calls it: host vectors in and out, walls and open sides, odd extents
        dict(name="euler_rhs_57x44x35_fp64", kind="euler_rhs", nx=57, ny=44, nz=35, prec="fp64", init="waves", bc="mixed", steps=1),
        # the headline run: 3D Euler, CWENO4 + Rusanov + SSPRK(4,3) in FP64 on 256^3
        dict(name="euler_256_fp64", kind="euler", nx=256, ny=256, nz=256, prec="fp64", init="pulse", bc="periodic", steps=1),
        # the double-float form on an ordinary grid with odd extents
        dict(name="euler_161x150x143_df64", kind="euler", nx=161, ny=150, nz=143, prec="df64", init="waves", bc="mixed", steps=2),
        # the FP32 form on the spherical blast, with the positivity fallback on as that run needs it
        dict(name="euler_blast_256_fp32", kind="euler", nx=256, ny=256, nz=256, prec="fp32", init="blast", bc="transmissive", steps=4),
        # Navier-Stokes: the Taylor-Green vortex (R4 values and gradients, viscous fluxes)
        dict(name="ns_tgv_96_fp64", kind="ns", nx=96, ny=96, nz=96, prec="fp64", init="tgv", bc="periodic", steps=2),
        # the acoustic finite-volume program between rigid walls
        dict(name="acoustic_200_fp64", kind="acoustic", nx=200, ny=200, nz=200, prec="fp64", init="waves", bc="adiabatic", steps=10),
        # 3D two-gas flow: the layered set-up of that program, a column of cells
        dict(name="mp3d_40x40x100_fp64", kind="mp3d", nx=40, ny=40, nz=100, prec="fp64", init="layers", bc="transmissive", steps=2),
        # 2D water-air bubble, Kapila model, FP32 reconstruction and flux
        dict(name="kapila_1024_fp32", kind="mp2d", nx=1024, ny=1024, nz=1, model=1, prec="fp32", init="bubble", bc="transmissive", steps=4),
        # the 2D bubble program's diffuse-interface model in FP64, odd extents
        dict(name="bubble_301x122_fp64", kind="mp2d", nx=301, ny=122, nz=1, model=0, prec="fp64", init="bubble", bc="mixed", steps=2),
        # the leapfrog acoustic solver: one grid that stays in L2
        dict(name="ctcs_512", kind="ctcs", nx=512, ny=512, nz=1, prec="fp64", init="gauss", bc="zero", steps=200),
        # many leapfrog instances of uneven size together
        dict(name="batch_48", kind="batch", nx=64, ny=768, nz=48, prec="fp64", init="gauss", bc="zero", steps=120),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["euler", "euler", "euler", "euler_rhs", "ns", "acoustic", "mp3d", "mp2d", "mp2d", "ctcs", "batch"])
    big = {"euler": 200, "euler_rhs": 80, "ns": 120, "acoustic": 220, "mp3d": 80}
    c = dict(kind=kind, prec="fp64", nz=1)
    if kind in big:
        n = _log(rng, 12, big[kind])
        c.update(nx=n, ny=max(8, int(n * rng.uniform(0.6, 1.2))), nz=max(8, int(n * rng.uniform(0.6, 1.2))))
    if kind in ("euler", "euler_rhs"):
        c.update(prec=rng.choice(["fp64", "fp64", "df64", "fp32"] if kind == "euler" else ["fp64", "df64"]),
                 init=rng.choice(["pulse", "waves"]), bc=rng.choice(["periodic", "mixed", "transmissive"]),
                 steps=rng.choice([1, 2, 4]) if kind == "euler" else 1)
    elif kind == "ns":
        c.update(prec=rng.choice(["fp64", "df64"]), init="tgv", bc="periodic", steps=rng.choice([1, 2, 4]))
        c.update(ny=c["nx"], nz=c["nx"])
    elif kind == "acoustic":
        c.update(prec=rng.choice(["fp64", "fp64", "df64"]), init="waves", bc=rng.choice(["periodic", "adiabatic"]), steps=rng.choice([4, 10, 16]))
    elif kind == "mp3d":
        c.update(init="layers", bc="transmissive", steps=rng.choice([1, 2]))
    elif kind == "mp2d":
        n = _log(rng, 40, 900)
        c.update(nx=n, ny=max(16, int(n * rng.uniform(0.5, 1.1))), model=rng.choice([0, 1]), prec=rng.choice(["fp64", "fp32"]),
                 init="bubble", bc=rng.choice(["transmissive", "mixed"]), steps=rng.choice([1, 2]))
    elif kind == "ctcs":
        n = _log(rng, 48, 1200)
        c.update(nx=n, ny=max(32, int(n * rng.uniform(0.5, 1.1))), init="gauss", bc=rng.choice(["zero", "periodic"]), steps=rng.choice([60, 100, 150]))
    else:  # nx..ny: the range of the instances' sides, nz: how many
        c.update(nx=64, ny=_log(rng, 128, 700), nz=rng.randrange(8, 64), init="gauss", bc="zero", steps=rng.choice([30, 90, 120]))
    return c


def _bc(c):
    return {"periodic": (PER,) * 6, "transmissive": (TRA,) * 6, "mixed": (TRA, REF, PER, PER, REF, TRA), "adiabatic": (ADI,) * 6}[c["bc"]]


def _bc2(c):
    return {"transmissive": (TRA,) * 4, "mixed": (TRA, TRA, REF, REF)}[c["bc"]]


# ------------------------------------------------------------------------------------------- initial states
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _axes(c, lo=0.0, h=None):
    """cell centres of z, y, x, shaped to broadcast over [z][y][x]"""
    h = 1.0 / c["nx"] if h is None else h
    a = [lo + (torch.arange(c[k], dtype=torch.float64, device=_dev()) + 0.5) * h for k in ("nz", "ny", "nx")]
    return a[0][:, None, None], a[1][None, :, None], a[2][None, None, :]


def _modes(c, rng, count=4):
    """a smooth field of size about one: seeded sine products over the box"""
    z, y, x = _axes(c)
    f = 0.0
    for _ in range(count):
        k, ph = rng.integers(1, 4, 3), rng.uniform(0, 2 * math.pi, 3)
        ly, lz = c["ny"] / c["nx"], c["nz"] / c["nx"]
        f = f + (rng.uniform(0.3, 1.0) * torch.sin(2 * math.pi * int(k[0]) * x + ph[0]) * torch.sin(2 * math.pi * int(k[1]) * y / ly + ph[1])) * torch.sin(
            2 * math.pi * int(k[2]) * z / lz + ph[2])
    return f / count


def _initial(c, seed):
    """the initial state [k][j][i][c] (or [j][i][c]) in FP64, from the seed alone"""
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    if kind in ("euler", "euler_rhs", "ns"):
        g1 = 0.4
        if c["init"] == "tgv":
            z, y, x = _axes(c, -math.pi, 2 * math.pi / c["nx"])
            ph = rng.uniform(0, 2 * math.pi, 3)
            x, y, z = x + ph[0], y + ph[1], z + ph[2]
            rho = torch.ones_like(x * y * z)
            u, v, w = torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z), 0.0 * rho
            p = 100 / 1.4 + (torch.cos(2 * z) + 2) * (torch.cos(2 * x) + torch.cos(2 * y) - 2) / 16
        elif c["init"] == "pulse":  # an acoustic pulse on a gas at rest
            z, y, x = _axes(c)
            m = rng.uniform(0.4, 0.6, 3)
            s = rng.uniform(0.04, 0.06) if c["nx"] >= 64 else rng.uniform(0.1, 0.14)
            r2 = (x - m[0]) ** 2 + (y - m[1] * c["ny"] / c["nx"]) ** 2 + (z - m[2] * c["nz"] / c["nx"]) ** 2
            dp = rng.uniform(0.8e-3, 1.2e-3) * torch.exp(-r2 / (2 * s * s))
            rho, p = 1 + dp, 1 / 1.4 + dp
            u = v = w = 0.0 * rho
        elif c["init"] == "blast":  # ten times the pressure in a sphere, one part in a thousand of noise
            z, y, x = _axes(c)
            m = rng.uniform(0.45, 0.55, 3)
            r2 = (x - m[0]) ** 2 + (y - m[1] * c["ny"] / c["nx"]) ** 2 + (z - m[2] * c["nz"] / c["nx"]) ** 2
            inside = r2 < 0.01
            gen = torch.Generator(device=_dev())
            gen.manual_seed(int(seed))
            noise = 2 * torch.rand(r2.shape, dtype=torch.float64, device=_dev(), generator=gen) - 1
            rho = torch.where(inside, 8.0, 1.0).to(torch.float64)
            p = torch.where(inside, 10 / 1.4, 1 / 1.4).to(torch.float64) * (1 + 1e-3 * noise)
            u = v = w = 0.0 * rho
        else:
            rho, p = 1 + 0.2 * _modes(c, rng), 1 / 1.4 + 0.1 * _modes(c, rng)
            u, v, w = (0.3 * _modes(c, rng) for _ in range(3))
        E = p / g1 + 0.5 * rho * (u * u + v * v + w * w)
        U = torch.stack([rho, rho * u, rho * v, rho * w, E], dim=-1)
    elif kind == "acoustic":
        U = torch.stack([_modes(c, rng), 0.5 * _modes(c, rng)], dim=-1)
    elif kind == "mp3d":
        z = _axes(c, -0.5, 1.0 / c["nz"])[0]
        step = lambda a: 0.5 * (1 + torch.tanh(a / 0.02))  # noqa: E731
        shock, gas = 1 - step(z + rng.uniform(0.22, 0.28)), step(z + 0.1) * (1 - step(z - 0.1))
        one = torch.ones(c["nz"], c["ny"], c["nx"], dtype=torch.float64, device=_dev())
        noise = 0.02 * _modes(c, rng)
        V = torch.stack([(1 + 0.3765 * shock - 0.862 * gas) * (one + noise), 0.05 * _modes(c, rng), 0.05 * _modes(c, rng), 0.3948 * shock * one + noise,
                         (1 + 0.57 * shock) * one, (1 - 0.999 * gas) * one])
        U = torch.movedim(_mp_cons(V, 3, 0, TWO_GASES), 0, -1)
    elif kind == "mp2d":  # an air bubble in water, a weak pressure step on its left
        _, y, x = _axes(c)
        y, x, h = y[0], x[0], 1.0 / c["nx"]
        m = rng.uniform(0.45, 0.55, 2)
        r = torch.sqrt((x - m[0]) ** 2 + (y - m[1] * c["ny"] / c["nx"]) ** 2)
        water = 1e-6 + (1 - 2e-6) * 0.5 * (1 + torch.tanh((r - 0.1 * rng.uniform(0.9, 1.1)) / (2 * h)))
        p = 1e5 + 9e5 * 0.5 * (1 - torch.tanh((x - 0.2) / (2 * h))) + 0 * r
        o = torch.ones_like(r)
        noise = [0.5 * _modes(dict(c, nz=1), rng)[0] for _ in range(2)]
        V = torch.stack([1000 * water + (1 - water), noise[0], noise[1], p, water] if c["model"] == 0 else [1000 * o, o, noise[0], noise[1], p, water])
        U = torch.movedim(_mp_cons(V, 2, c["model"], WATER_AIR), 0, -1)
    return np.ascontiguousarray(U.cpu().numpy())


def _ctcs_levels(c, seed):
    rng = np.random.default_rng(seed)
    h = 2.0 / c["nx"]
    x, y = -1 + np.arange(c["nx"]) * h, -1 + np.arange(c["ny"]) * h
    m, s = rng.uniform(-0.2, 0.2, 2), rng.uniform(0.04, 0.08)
    p0 = np.exp(-((x[None, :] - m[0]) ** 2 + (y[:, None] + 1 - c["ny"] / c["nx"] - m[1]) ** 2) / (2 * s * s))
    return p0, 0.999 * p0, 0.5


def _instances(c, seed):
    rng = np.random.default_rng(c["nx"] * 1000003 + c["ny"] * 101 + c["nz"])  # the sizes go with the case, the sources with the seed
    sides = np.exp(rng.uniform(math.log(c["nx"]), math.log(c["ny"]), (c["nz"], 2)))
    rng = np.random.default_rng(seed)
    out = []
    for n, m in np.rint(sides).astype(int):
        n, h = int(n), 2.0 / int(n)
        xs, ys = rng.uniform(-0.8, 0.8, 2)
        out.append(dict(nx=n, ny=max(32, min(int(m), 2 * n)), xmin=-1.0, ymin=-1.0, h=h, c0=1.0, dt=0.5 * h, xs=float(xs), ys=float(ys),
                        sigma=float(rng.uniform(0.02, 0.1)), freq=float(1 / (rng.uniform(8, 32) * h))))
    return out


# ------------------------------------------------------------------------------------------ prepare and run
class State:
    """a solver handle, its initial state and how far its run is"""


def _euler_ctx(c):
    prec = {"fp64": FP64, "fp32": FP32, "df64": DF64}[c["prec"]]
    ns = c["kind"] == "ns"
    return H.AppCtx(N_x=c["nx"], N_y=c["ny"], N_z=c["nz"], h=(2 * math.pi if ns else 1.0) / c["nx"], CFL=0.6 if ns else 0.4, boundaries=_bc(c),
                    recon=L.RECON_LINEAR4 if ns else L.RECON_CWENO4, precision=prec, positivity=int(c["init"] == "blast"), mu=0.01 if ns else 0.0)


def prepare(case, seed):
    c, s = case, State()
    s.case, s.kind, s.steps, s.done, s.horizon = c, c["kind"], c["steps"], 0, {"ctcs": 4000, "acoustic": 4000, "mp2d": 120, "mp3d": 40}.get(c["kind"], 400)
    if s.kind == "ctcs":
        p0, p1, alpha = _ctcs_levels(c, seed)
        h = 2.0 / c["nx"]
        s.levels = (p0, p1)
        s.solver = H.Leapfrog(p0.shape, dx=h, dt=alpha * h, c0=1.0, form=0, bc=ZERO if c["bc"] == "zero" else PER)
    elif s.kind == "batch":
        s.solver = H.BatchLeapfrog([H.Monopole(**m) for m in _instances(c, seed)], tile=(32, 64))
        s.solver.set_classes(1)
    else:
        s.U = _initial(c, seed)
        if s.kind in ("euler", "euler_rhs", "ns"):
            s.solver = H.EulerSolver(_euler_ctx(c))
        elif s.kind == "acoustic":
            s.solver = H.AcousticFV3D(c["nx"], c["ny"], c["nz"], 1.0 / c["nx"], 0.3 / c["nx"], boundaries=_bc(c), precision=DF64 if c["prec"] == "df64" else FP64)
        elif s.kind == "mp3d":
            s.solver = H.Multiphase3D(c["nx"], c["ny"], c["nz"], 1.0 / c["nz"], CFL=0.6, boundaries=_bc(c), eos=TWO_GASES, mu=(0.0, 0.0))
        else:
            s.solver = H.Multiphase2D(c["nx"], c["ny"], 1.0 / c["nx"], CFL=0.6, boundaries=_bc2(c), model=c["model"], eos=WATER_AIR,
                                      precision=FP32 if c["prec"] == "fp32" else FP64)
    if s.kind != "euler_rhs":
        _start(s)
    return s


def _start(s):
    if s.kind == "ctcs":
        s.solver.set(*s.levels)
    elif s.kind == "batch":
        for q, m in enumerate(s.solver.instances):
            zero = np.zeros((m.ny, m.nx))
            s.solver.set(q, zero, zero)
    else:
        s.solver.set_state(s.U)
        s.solver.t = s.solver.next_dt = 0.0
    s.done = 0


class _DeviceState:
    """the solver's resident state as torch sees it (no copy)"""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def run(s):
    if s.kind == "euler_rhs":
        rhs = s.solver.RHSFunction(0.0, s.U)
        return {"rhs": rhs, "dt": s.solver.ctx.dt}
    if s.done + s.steps > s.horizon and s.kind != "batch":
        _start(s)
    s.done += s.steps
    if s.kind == "ctcs":
        s.solver.UpdatePressure(s.steps)
        old, new = s.solver.get()
        return {"p_old": old, "p": new}
    if s.kind == "batch":
        s.solver.step(s.steps)
        return [s.solver.get(q)[1] for q in range(len(s.solver.instances))]
    s.solver.step(s.steps)
    if s.kind in ("euler", "ns"):
        c = s.case
        held = _DeviceState(s.solver.device_state_ptr(), (5, c["nz"], c["ny"], c["nx"]), s.solver)
        return {"state": torch.as_tensor(held, device="cuda"), "t": s.solver.t, "next_dt": s.solver.next_dt}
    if s.kind == "acoustic":
        return {"state": s.solver.get_state()}
    return {"state": s.solver.get_state(), "t": s.solver.t, "next_dt": s.solver.next_dt}


def work(case):
    """bytes: the state read and written once; flops: the operations of the scheme per cell and stage (counted on
    the reconstruction, the face solves and the update), times cells, stages and steps"""
    c = case
    n, stages = c["nx"] * c["ny"] * c["nz"], 4 * c["steps"]
    kind = c["kind"]
    if kind == "batch":
        inst = _instances(c, 0)
        n = sum(m["nx"] * m["ny"] for m in inst)
        return {"bytes": 8.0 * n * 4, "flops": 9.0 * n * c["steps"]}
    if kind == "ctcs":
        return {"bytes": 8.0 * n * 4, "flops": 8.0 * n * c["steps"]}
    if kind == "euler_rhs":
        return {"bytes": 80.0 * n, "flops": 4600.0 * n}
    nv, flops = {"euler": (5, 4600.0), "ns": (5, 6600.0), "acoustic": (2, 60.0), "mp3d": (6, 11000.0), "mp2d": (6, 2400.0)}[kind]
    return {"bytes": 16.0 * nv * n, "flops": flops * n * stages}


# ------------------------------------------------------------------- the same results in plain 64-bit tensors
def _ghosts(S, bc, flip):
    """S [c][...][y][x] with three ghost layers; flip(axis from x) = the components negated at its walls"""
    nd = S.dim() - 1
    for ax in range(nd):
        dim, n = nd - ax, S.shape[nd - ax]
        i = torch.arange(-3, n + 3, device=S.device)
        lo, hi = bc[2 * ax], bc[2 * ax + 1]
        j = torch.where(i < 0, {PER: i + n, TRA: 0 * i}.get(lo, -1 - i), torch.where(i >= n, {PER: i - n, TRA: 0 * i + n - 1}.get(hi, 2 * n - 1 - i), i))
        S = S.index_select(dim, j.clamp(0, n - 1))
        sign = torch.ones(n + 6, dtype=S.dtype, device=S.device)
        if lo in (REF, ADI):
            sign[:3] = -1
        if hi in (REF, ADI):
            sign[-3:] = -1
        shape = [1] * nd
        shape[dim - 1] = n + 6
        for comp in flip(ax):
            S[comp] *= sign.reshape(shape)
    return S


def _at(G):
    """value of a ghosted field at an offset from every cell of the box widened by one"""
    nd = G.dim()

    def at(*o):  # offsets along x, y(, z)
        return G[tuple(slice(2 + o[nd - 1 - d], G.shape[d] - 2 + o[nd - 1 - d]) for d in range(nd))]

    return at


def _unit(nd, *steps):
    o = [0] * nd
    for axis, k in steps:
        o[axis] += k
    return o


def _cweno(G, linear=False):
    """the polynomial coefficients {(exponents): value} of weno() on every cell of the widened box, and the cell value"""
    at, nd = _at(G), G.dim()
    e = lambda *s: at(*_unit(nd, *s))  # noqa: E731
    u0, ax = e(), range(nd)
    pairs = [(a, b) for a in ax for b in ax if a < b]
    d4 = [(11 * e((a, -2)) - 82 * e((a, -1)) + 82 * e((a, 1)) - 11 * e((a, 2))) / 120 for a in ax]
    dd4 = [(e((a, -1)) - 2 * u0 + e((a, 1))) / 2 for a in ax]
    ddd4 = [(-e((a, -2)) + 2 * (e((a, -1)) - e((a, 1))) + e((a, 2))) / 12 for a in ax]
    q = {(a, b, s, t): e((a, s), (b, t)) for a, b in pairs for s in (-1, 1) for t in (-1, 1)}
    x4 = {(a, b): (q[a, b, -1, -1] - q[a, b, -1, 1] - q[a, b, 1, -1] + q[a, b, 1, 1]) / 4 for a, b in pairs}
    aab = {(a, b): (-q[a, b, -1, -1] + q[a, b, -1, 1] - q[a, b, 1, -1] + q[a, b, 1, 1]) / 4 + (e((b, -1)) - e((b, 1))) / 2 for a, b in pairs}
    abb = {(a, b): (e((a, -1)) - e((a, 1))) / 2 + (q[a, b, 1, 1] - q[a, b, -1, -1] - q[a, b, -1, 1] + q[a, b, 1, -1]) / 4 for a, b in pairs}
    xyz = None
    if nd == 3:
        xyz = sum(s * t * r * e((0, s), (1, t), (2, r)) for s in (-1, 1) for t in (-1, 1) for r in (-1, 1)) / 8
    if linear:
        lin, quad, cross, wr = d4, dd4, x4, 1.0
    else:
        cube = 39.06 if nd == 3 else 39.05
        if nd == 3:
            IS4 = sum(d4[a] ** 2 + 0.2 * d4[a] * ddd4[a] for a in ax) + 61 / 48 * xyz**2
        else:
            IS4 = sum((d4[a] + 0.1 * ddd4[a]) ** 2 for a in ax)
        IS4 = IS4 + 13 / 3 * sum(v * v for v in dd4) + 7 / 6 * sum(v * v for v in x4.values()) + cube * sum(v * v for v in ddd4)
        IS4 = IS4 + 4.7 * (sum(v * v for v in aab.values()) + sum(v * v for v in abb.values()))
        c1 = [(e((a, 1)) - e((a, -1))) / 2 for a in ax]
        subs = [(c1, dd4, x4)]
        for a in ax:
            for s in (1, -1):
                d, dd, x = list(c1), list(dd4), dict(x4)
                d[a] = s * (-1.5 * u0 + 2 * e((a, s)) - 0.5 * e((a, 2 * s)))
                dd[a] = (u0 - 2 * e((a, s)) + e((a, 2 * s))) / 2
                for b in ax:
                    if b != a:
                        x[min(a, b), max(a, b)] = s * ((e((a, s), (b, 1)) - e((a, s), (b, -1))) / 2 - c1[b])
                subs.append((d, dd, x))
        gam = 0.85
        g3 = [(1 - gam) * gam] + [(1 - gam) ** 2 / (2 * nd)] * (2 * nd)
        IS3 = [sum(v * v for v in d) + 13 / 3 * sum(v * v for v in dd) + 7 / 6 * sum(v * v for v in x.values()) for d, dd, x in subs]
        w4 = gam / (IS4 + 1e-12) ** 4
        w3 = [g / (v + 1e-12) ** 4 for g, v in zip(g3, IS3)]
        total = w4 + sum(w3)
        w4, w3 = w4 / total, [w / total for w in w3]
        wr = w4 / gam
        mix = lambda hi, lo: wr * (hi - sum(g * v for g, v in zip(g3, lo))) + sum(w * v for w, v in zip(w3, lo))  # noqa: E731
        lin = [mix(d4[a], [m[0][a] for m in subs]) for a in ax]
        quad = [mix(dd4[a], [m[1][a] for m in subs]) for a in ax]
        cross = {k: mix(x4[k], [m[2][k] for m in subs]) for k in pairs}
    cf = {}
    ex = lambda *s: tuple(_unit(nd, *s))  # noqa: E731
    for a in ax:
        cf[ex((a, 1))], cf[ex((a, 2))], cf[ex((a, 3))] = lin[a], quad[a], wr * ddd4[a]
    for a, b in pairs:
        cf[ex((a, 1), (b, 1))] = cross[a, b]
        cf[ex((a, 2), (b, 1))], cf[ex((a, 1), (b, 2))] = wr * aab[a, b], wr * abb[a, b]
    if nd == 3:
        cf[1, 1, 1] = wr * xyz
    return u0, cf


_B = {0: lambda t: 1.0, 1: lambda t: t, 2: lambda t: t * t - 1 / 12, 3: lambda t: t * (t * t - 3 / 20)}
_DB = {0: lambda t: 0.0, 1: lambda t: 1.0, 2: lambda t: 2 * t, 3: lambda t: 3 * t * t - 3 / 20}


def _value(poly, pt, deriv=None):
    u0, cf = poly
    v = u0.clone() if deriv is None else torch.zeros_like(u0)
    for ex, k in cf.items():
        b = 1.0
        for a, (n, t) in enumerate(zip(ex, pt)):
            b *= (_DB if a == deriv else _B)[n](t)
        if b:
            v += k * b
    return v


def _face_points(nd, a, side):
    others = [b for b in range(nd) if b != a]
    for q in range(2 ** (nd - 1)):
        pt = [0.0] * nd
        pt[a] = side * 0.5
        for m, b in enumerate(others):
            pt[b] = GP if (q >> (len(others) - 1 - m)) & 1 else -GP
        yield tuple(pt)


def _sides(T, a, nd):
    """(left, right) values of the faces normal to axis a from per-cell traces (high side, low side) on the widened box"""
    hi, lo = T
    left, right = [], []
    for d in range(nd):
        axis = nd - 1 - d
        n = hi.shape[hi.dim() - nd + d]
        left.append(slice(0, n - 1) if axis == a else slice(1, n - 1))
        right.append(slice(1, n) if axis == a else slice(1, n - 1))
    lead = (slice(None),) * (hi.dim() - nd)
    return hi[lead + tuple(left)], lo[lead + tuple(right)]


def _diff(F, a, nd):
    dim = F.dim() - 1 - a
    n = F.shape[dim]
    return F.narrow(dim, 1, n - 1) - F.narrow(dim, 0, n - 1)


def _euler_rhs(S, c, h, mu, linear, positivity):
    G = _ghosts(S, _bc(c), lambda ax: (1 + ax,))
    polys = [_cweno(G[q], linear) for q in range(5)]
    gam, smax, svis = 1.4, 0.0, 0.0
    if positivity:
        ok = torch.ones_like(polys[0][0], dtype=torch.bool)
        for a in range(3):
            for side in (-1, 1):
                for pt in _face_points(3, a, side):
                    Q = [_value(p, pt) for p in polys]
                    ok &= (Q[0] >= 1e-14) & (0.4 * (Q[4] - 0.5 * (Q[1] ** 2 + Q[2] ** 2 + Q[3] ** 2) / Q[0]) >= 1e-12)
        polys = [(u0, {k: torch.where(ok, v, 0.0) for k, v in cf.items()}) for u0, cf in polys]
    R = torch.zeros_like(S)
    for a in range(3):
        F = 0.0
        for hi, lo in zip(_face_points(3, a, 1), _face_points(3, a, -1)):
            sides = _sides((torch.stack([_value(p, hi) for p in polys]), torch.stack([_value(p, lo) for p in polys])), a, 3)
            fl, sp = [], []
            for Q in sides:
                u = Q[1:4] / Q[0]
                p = 0.4 * (Q[4] - 0.5 * Q[0] * (u * u).sum(0))
                f = Q * u[a]
                f[1 + a] += p
                f[4] += p * u[a]
                fl.append(f)
                sp.append(u[a].abs() + torch.sqrt(gam * p / Q[0]))
            s = torch.maximum(*sp)
            smax = max(smax, float(s.max()))
            f = 0.5 * (fl[0] + fl[1] - s * (sides[1] - sides[0]))
            if mu:
                grads = [[torch.stack([_value(p, pt, b) for p in polys]) / h for b in range(3)] for pt in (hi, lo)]
                k = 2.5 * mu * gam
                for Q, g in zip(sides, zip(*[_sides((grads[0][b], grads[1][b]), a, 3) for b in range(3)])):
                    r, u = Q[0], Q[1:4] / Q[0]
                    du = [g[b][1:4] - u * g[b][0] / r for b in range(3)]
                    m2 = (Q[1:4] ** 2).sum(0)
                    dT = [-0.4 * g[b][0] / r**2 * (Q[4] - 0.5 * m2 / r) + 0.4 / r * (g[b][4] - (Q[1:4] * g[b][1:4]).sum(0) / r + 0.5 * m2 * g[b][0] / r**2) for b in range(3)]
                    div = -2 / 3 * mu * (du[0][0] + du[1][1] + du[2][2])
                    tau = [mu * (du[a][b] + du[b][a]) + (div if a == b else 0.0) for b in range(3)]
                    for b in range(3):
                        f[1 + b] -= 0.5 * tau[b]
                    f[4] -= 0.5 * (sum(u[b] * tau[b] for b in range(3)) + k * dT[a])
                    svis = max(svis, float((max(4 / 3, gam) * mu / r).max()))
            F = F + 0.25 * f
        R -= _diff(F, a, 3) / h
    return R, (smax, svis)


def _acoustic_rhs(S, c, h):
    G = _ghosts(S[:1], _bc(c), lambda ax: (0,))[0]
    poly = _cweno(G, True)
    div = 0.0
    for a in range(3):
        F = 0.0
        for hi, lo in zip(_face_points(3, a, 1), _face_points(3, a, -1)):
            gl, gr = _sides((_value(poly, hi, a), _value(poly, lo, a)), a, 3)
            F = F + 0.125 * (gl + gr)
        div = div + _diff(F, a, 3) / (h * h)
    return torch.stack([S[1], div])


def _mix(eos, a):
    """gamma and stiffness of the mixture (phase 1 fraction a)"""
    g1, p1, g2, p2 = eos
    g = 1 + (g1 - 1) * (g2 - 1) / ((1 - a) * (g1 - 1) + a * (g2 - 1))
    return g, (g - 1) / g * (g1 * p1 * a / (g1 - 1) + g2 * p2 * (1 - a) / (g2 - 1))


def _mp_parts(V, nd, model):
    """density, velocities, pressure, fraction of primitive variables"""
    if model == 0:
        return V[0], V[1 : 1 + nd], V[1 + nd], V[2 + nd]
    return V[5] * V[0] + (1 - V[5]) * V[1], V[2:4], V[4], V[5]


def _mp_cons(V, nd, model, eos):
    r, u, p, a = _mp_parts(V, nd, model)
    g, pi = _mix(eos, a)
    E = (p + g * pi) / (g - 1) + 0.5 * r * (u * u).sum(0)
    return torch.stack([*([r] if model == 0 else [a * V[0], (1 - a) * V[1]]), *(r * u), E, a])


def _mp_prim(Q, nd, model, eos):
    k = 1 if model == 0 else 2
    r, a = (Q[0] if model == 0 else Q[0] + Q[1]), Q[-1]
    g, pi = _mix(eos, a)
    u = Q[k : k + nd] / r
    p = (g - 1) * (Q[k + nd] - 0.5 * r * (u * u).sum(0)) - g * pi
    return torch.stack([*([r] if model == 0 else [Q[0] / a, Q[1] / (1 - a)]), *u, p, a])


def _hllc(V, n, nd, model, eos):
    """the flux along n with the interface velocity appended, and the largest speed"""
    side = []
    for v in V:
        r, u, p, a = _mp_parts(v, nd, model)
        g, pi = _mix(eos, a)
        Q, un = _mp_cons(v, nd, model, eos), (u * n).sum(0)
        F = Q * un
        k = 1 if model == 0 else 2
        F[k : k + nd] += p * n
        F[k + nd] += p * un
        side.append((r, u, p, Q, un, torch.cat([F, un[None]]), torch.sqrt(g * (p + pi) / r)))
    (rL, uL, pL, QL, nL, FL, cL), (rR, uR, pR, QR, nR, FR, cR) = side
    SL, SR = torch.minimum(nR - cR, nL - cL), torch.maximum(nL + cL, nR + cR)
    mL, mR = rL * (SL - nL), rR * (SR - nR)
    Ss = (pR - pL + nL * mL - nR * mR) / (mL - mR)
    star = []
    for (r, u, p, Q, un, F, _), S in zip(side, (SL, SR)):
        f = (S - un) / (S - Ss)
        k = 1 if model == 0 else 2
        Us = Q * f
        Us[k : k + nd] = r * f * (u + (Ss - un) * _frame_normal(n, nd))
        Us[k + nd] = r * f * (Q[k + nd] / r + (Ss - un) * (Ss + p / (r * (S - un))))
        star.append(torch.cat([F[:-1] + S * (Us - Q), (un + S * (f - 1))[None]]))
    F = torch.where(SL > 0, FL, torch.where(Ss >= 0, star[0], torch.where(SR >= 0, star[1], FR)))
    return F, torch.maximum(nL.abs() + cL, nR.abs() + cR)


def _tangents(n, w):
    """the solver's two tangents; its inner and its rotated form differ in what w is"""
    x, y, z = n
    first = (y + z).abs() > (y - z).abs()
    l1, l2 = torch.sqrt(2 * (1 + z * (y - x) + x * y)), torch.sqrt(2 * (1 - x * y - x * z - y * z))
    t1 = torch.where(first, torch.stack([y + z, z - x, -(x + y)]) / l1, torch.stack([y - z, z - x, x - y]) / l2)
    a = torch.stack([x * (z - y) - y * y - z * z, y * (x + z) + x * x + z * z, z * (x - w) - x * x - y * y]) / l1
    b = torch.stack([x * (y + z) - y * y - z * z, y * (x + z) - x * x - z * z, z * (x + y) - x * x - y * y]) / l2
    return t1, torch.where(first, a, b)


def _frame_normal(n, nd):
    """what the star state's normal velocity multiplies: the first column of the inverse of the solver's frame"""
    if nd == 2:
        return n
    t1, t2 = _tangents(n, n[2])
    c = torch.linalg.cross(t1, t2, dim=0)
    return c / (n * c).sum(0)


def _rot_hllc(V, a, nd, model, eos):
    du = _mp_parts(V[1], nd, model)[1] - _mp_parts(V[0], nd, model)[1]
    dq = torch.sqrt((du * du).sum(0))
    e = torch.zeros_like(du)
    e[a] = 1
    n = torch.where(dq < 1e-10, e, du / dq)
    n = torch.where(n[a] < 0, -n, n)
    frame = [n, torch.stack([-n[1], n[0]])] if nd == 2 else [n, *_tangents(n, n[1])]
    F = smax = 0.0
    for m in frame:
        m = torch.where(m[a] < 0, -m, m)
        f, s = _hllc(V, m, nd, model, eos)
        F, smax = F + m[a] * f, max(smax, float(s.max()))
    return F, smax


def _nodes(nd):
    if nd == 2:
        return [p for a in range(2) for s in (-1, 1) for p in _face_points(2, a, s)]
    pts = [(0.0, 0.0, 0.0)] + [tuple(k * t for t in _unit(3, (a, 1))) for a in range(3) for k in (0.5, 0.25, -0.25, -0.5)]
    h = (-0.5, 0.0, 0.5)
    return pts + [(x, y, z) for x in h for y in h for z in h if (x != 0) + (y != 0) + (z != 0) >= 2]


def _mp_rhs(S, c, nd, model, eos, h):
    bc = _bc(c) if nd == 3 else _bc2(c)
    k = 1 if model == 0 else 2
    P = _mp_prim(S, nd, model, eos)
    G = _ghosts(P, bc, lambda ax: (k + ax,))
    polys = [_cweno(G[q]) for q in range(len(P))]
    ok = torch.ones_like(polys[0][0], dtype=torch.bool)
    for pt in _nodes(nd):
        V = [_value(p, pt) for p in polys]
        ok &= (V[0] >= 1e-14) & (V[k + nd] + _mix(eos, V[-1])[1] >= 1e-12)
        if nd == 2:
            ok &= (V[-1] >= 0) & (V[-1] <= 1) & ((V[1] >= 1e-14) if model == 1 else True)
    for q, (u0, cf) in enumerate(polys):
        low = {}
        if nd == 2:  # the two-dimensional programs keep a limited slope
            at = _at(G[q])
            for a in range(2):
                p, m = at(*_unit(2, (a, 1))) - u0, u0 - at(*_unit(2, (a, -1)))
                low[tuple(_unit(2, (a, 1)))] = torch.where(p * m < 0, 0.0, torch.where(p.abs() < m.abs(), p, m))
        polys[q] = (u0, {ex: torch.where(ok, v, low.get(ex, torch.zeros_like(v))) for ex, v in cf.items()})
    R, smax = torch.zeros_like(S), 0.0
    for a in range(nd):
        F, w = 0.0, 0.5 ** (nd - 1)
        for hi, lo in zip(_face_points(nd, a, 1), _face_points(nd, a, -1)):
            f, s = _rot_hllc(_sides((torch.stack([_value(p, hi) for p in polys]), torch.stack([_value(p, lo) for p in polys])), a, nd), a, nd, model, eos)
            F, smax = F + w * f, max(smax, s)
        d = _diff(F, a, nd)
        R -= d[:-1] / h
        R[-1] += P[-1] * d[-1] / h
    return R, (smax, 0.0)


def _ssp43(S, rhs, dt_of, steps, fixed=None):
    t, dt = 0.0, fixed
    for _ in range(steps):
        R, s = rhs(S)
        dt = dt_of(s) if dt is None else dt
        W = S + dt / 2 * R
        W = W + dt / 2 * rhs(W)[0]
        W = 2 / 3 * S + dt / 6 * rhs(W)[0] + W / 3
        R, s = rhs(W)
        S, t = W + dt / 2 * R, t + dt
        dt = dt_of(s) if fixed is None else fixed
    return S, t, dt


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "ctcs":
        p0, p1, alpha = _ctcs_levels(c, seed)
        a, b = torch.from_numpy(p0).to(_dev()), torch.from_numpy(p1).to(_dev())
        for _ in range(c["steps"]):
            z = torch.nn.functional.pad(b[None, None], (1, 1, 1, 1), mode="circular" if c["bc"] == "periodic" else "constant")[0, 0]
            a, b = b, alpha**2 * (z[2:, 1:-1] + z[:-2, 1:-1] + z[1:-1, 2:] + z[1:-1, :-2] - 4 * b) + 2 * b - a
        return {"p_old": a.cpu().numpy(), "p": b.cpu().numpy()}
    if kind == "batch":
        out = []
        for m in _instances(c, seed):
            x = m["xmin"] + torch.arange(m["nx"], dtype=torch.float64, device=_dev()) * m["h"]
            y = m["ymin"] + torch.arange(m["ny"], dtype=torch.float64, device=_dev()) * m["h"]
            src = torch.exp(-((x[None, :] - m["xs"]) ** 2 + (y[:, None] - m["ys"]) ** 2) / (2 * m["sigma"] ** 2))
            a = torch.zeros_like(src)
            b, k2 = a.clone(), (m["c0"] * m["dt"]) ** 2
            for s in range(c["steps"]):
                z = torch.nn.functional.pad(b, (1, 1, 1, 1))
                lap = (z[2:, 1:-1] + z[:-2, 1:-1] + z[1:-1, 2:] + z[1:-1, :-2] - 4 * b) / m["h"] ** 2
                a, b = b, 2 * b - a + k2 * lap + k2 * math.sin(2 * math.pi * m["freq"] * s * m["dt"]) * src
            out.append(b.cpu().numpy())
        return out
    S = torch.from_numpy(_initial(c, seed)).to(_dev())
    nd = S.dim() - 1
    S = torch.movedim(S, -1, 0).contiguous()
    h = 1.0 / c["nx"]
    if kind in ("euler", "euler_rhs", "ns"):
        ctx = _euler_ctx(c)
        h = ctx.h
        rhs = lambda W: _euler_rhs(W, c, h, ctx.mu, ctx.recon == L.RECON_LINEAR4, ctx.positivity)  # noqa: E731
        dt_of = lambda s: ctx.CFL * h / 3 / (s[0] + 2 * s[1] / h)  # noqa: E731
        if kind == "euler_rhs":
            R, s = rhs(S)
            return {"rhs": torch.movedim(R, 0, -1).contiguous().cpu().numpy(), "dt": dt_of(s)}
        S, t, dt = _ssp43(S, rhs, dt_of, c["steps"])
        return {"state": S, "t": t, "next_dt": dt}
    if kind == "acoustic":
        S, _, _ = _ssp43(S, lambda W: (_acoustic_rhs(W, c, h), None), None, c["steps"], fixed=0.3 / c["nx"])
        return {"state": torch.movedim(S, 0, -1).contiguous().cpu().numpy()}
    if kind == "mp3d":
        h = 1.0 / c["nz"]
        S, t, dt = _ssp43(S, lambda W: _mp_rhs(W, c, nd, 0, TWO_GASES, h), lambda s: 0.6 * h / 3 / s[0], c["steps"])
    else:
        S, t, dt = _ssp43(S, lambda W: _mp_rhs(W, c, nd, c["model"], WATER_AIR, h), lambda s: 0.6 * h / 2 / s[0], c["steps"])
    return {"state": torch.movedim(S, 0, -1).contiguous().cpu().numpy(), "t": t, "next_dt": dt}
