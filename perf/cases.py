"""The work that is measured: whole calls of the solver as its users make them.

A case is a dict of plain values.  ``kind`` names the call:

* ``step``      a state into the handle, SSPRK(5,2) steps, the state back out
* ``rhs``       one right-hand side of a device tensor (the sub-solver's ``step``)
* ``gradient``  a fixed-step trajectory with checkpoints and its discrete adjoint
* ``jacobian``  one tangent and one adjoint right-hand side (Newton-Krylov, sensitivities)
* ``ensemble``  a batch of independent meshes of orders 2..5, one step each

and ``problem`` the equation, mesh and boundaries (``n`` is the vertex grid of a
jittered square, so K = 2 (n-1)^2 triangles; ``N`` the polynomial order):

* ``advection``  periodic unit square, scalar advection
* ``vortex``     periodic [0,10]^2, Euler in 4 fields, Lax-Friedrichs flux
* ``channel``    [0,2] x [0,1], Euler in 5 (or 4) fields, wall, outflow, inflow and
                 Dirichlet sides, HLL flux; with ``limiter`` Apollo's Euler limiter
* ``cavity``     unit square with conducting walls, transverse-magnetic Maxwell (3 fields)
* ``cleaning``   unit square with conducting walls, the 8-field Maxwell system with
                 divergence cleaning and a volume current source

Sizes come from this repository's configurations (K = 1,922 advection, K = 130,050
vortex, K = 522,242 cavity, the K = 32,258 adjoint) and from meshes between them.
"""
import functools
import math
import os
import re

import numpy as np
import torch
import torch.utils.checkpoint

from apollo_b200 import NodalDG2d, NodalDG2dBatch
from apollo_b200.mesh import jittered_square

CFL = 0.5
FIELDS = {"advection": 1, "vortex": 4, "channel": 5, "cavity": 3, "cleaning": 8}
# Mach_number, Flow_angle, gas_gamma, Pressure, density / density, velocities, gas_gamma, pressure
INFLOW = (0.4, -60.0, 1.4, 1.0, 1.0)
DIRICHLET = (1.0, 0.5, 0.0, 0.0, 1.4, 1.0)


def listed():
    return [
        # the smallest mesh in use: ten launch-bound steps of the advection configuration
        dict(name="advection_small", kind="step", problem="advection", N=3, n=32, steps=10, precision="fp64"),
        # a low-order run on a mesh of middling size (K = 18,432)
        dict(name="vortex_N2", kind="step", problem="vortex", N=2, n=97, steps=3, precision="fp64"),
        # the headline configuration (K = 130,050, N = 4) in both arithmetics
        dict(name="vortex_N4", kind="step", problem="vortex", N=4, n=256, steps=2, precision="fp64"),
        dict(name="vortex_N4_mixed", kind="step", problem="vortex", N=4, n=256, steps=2, precision="mixed"),
        # the largest configuration: the order-5 cavity on its own mesh (K = 522,242)
        dict(name="cavity_N5", kind="step", problem="cavity", N=5, n=512, steps=1, precision="fp64"),
        # the same cavity in mixed precision on an odd mesh (K = 66,978)
        dict(name="cavity_N5_mixed", kind="step", problem="cavity", N=5, n=184, steps=2, precision="mixed"),
        # a single right-hand side, as Apollo's own time integrator calls it: all four
        # boundary kinds, the HLL flux, 5 fields, K = 28,800
        dict(name="channel_rhs", kind="rhs", problem="channel", N=3, n=121, precision="fp64"),
        # a limited run of the channel (Apollo's forward-facing-step setting), K = 8,192
        dict(name="channel_limited", kind="step", problem="channel", N=3, n=65, steps=2, precision="fp64",
             limiter=True),
        # the 8-field system with sources, K = 14,450
        dict(name="cleaning_N4", kind="step", problem="cleaning", N=4, n=86, steps=2, precision="fp64"),
        # the adjoint configuration's mesh and order (K = 32,258), ten steps, checkpoints every five
        dict(name="gradient", kind="gradient", problem="vortex", N=3, n=128, steps=10, every=5),
        # one Jacobian product each way, K = 16,200
        dict(name="jacobian", kind="jacobian", problem="vortex", N=4, n=91),
        # an ensemble of small and medium vortices, orders 2..5 in turn
        dict(name="ensemble", kind="ensemble", problem="vortex", count=12, kmin=1500, kmax=16000, precision="fp64"),
    ]


def draw(rng):
    def grid(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step"] * 6 + ["rhs"] * 2 + ["gradient", "jacobian", "ensemble"])
    if kind == "ensemble":
        kmin = grid(500, 4000)
        return dict(kind=kind, problem="vortex", count=rng.randint(3, 14), kmin=kmin, kmax=kmin * rng.randint(2, 8),
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "gradient":
        return dict(kind=kind, problem="vortex", N=rng.randint(2, 4), n=grid(24, 140), steps=rng.randint(4, 10),
                    every=rng.randint(2, 5))
    if kind == "jacobian":
        return dict(kind=kind, problem=rng.choice(["vortex", "cavity"]), N=rng.randint(2, 5), n=grid(20, 180))
    problem = rng.choice(["advection", "vortex", "vortex", "channel", "cavity", "cleaning"])
    N = rng.randint(2, 5)
    top = {"advection": 320, "vortex": 260, "channel": 200, "cavity": 320, "cleaning": 150}[problem]
    case = dict(kind=kind, problem=problem, N=N, n=grid(16, top), precision=rng.choice(["fp64", "fp64", "fp64", "mixed"]))
    if kind == "step":
        case["steps"] = rng.randint(1, 4)
        if problem == "channel" and N <= 4 and rng.random() < 0.5:
            case["limiter"] = True
    return case


# ---------------------------------------------------------------- inputs ----
def channel_bcs():
    return (("eulerWallBC", ()), ("eulerZeroGradientBC", ()), ("eulerInflowBC", INFLOW), ("eulerDirichletBC", DIRICHLET))


def equation(problem):
    """(kind, parameters, boundary conditions, sources, numerical flux) of a problem."""
    return {
        "advection": ("advectionEqn", (1.0, 0.5, 0.0), (), (), "LF"),
        "vortex": ("eulerEqn2d", (1.4, 0.0, 0.0), (), (), "LF"),
        "channel": ("eulerEqn", (1.4, 0.0, 0.0), channel_bcs(), (), "HLL"),
        "cavity": ("maxwellTM", (1.0,), (("maxwellTransverseMagneticBC", ()),), (), "LF"),
        "cleaning": ("phMaxwellEqn", (1.0, 0.8, 0.6), (("phmConductingWallBC", ()),),
                     (("tranverseMagneticSrc", (2,), ()),), "LF"),
    }[problem]


@functools.lru_cache(maxsize=32)
def mesh_of(problem, n, seed=0):
    """The mesh a user reads once; cases of one size share it."""
    if problem == "advection":
        return jittered_square(n, seed=seed)
    if problem == "vortex":
        return jittered_square(n, (0.0, 0.0), (10.0, 10.0), seed=seed)
    if problem != "channel":
        return jittered_square(n, seed=seed, periodic=False)
    mesh = jittered_square(n, (0.0, 0.0), (2.0, 1.0), seed=seed, periodic=False)
    for f, (i, j) in enumerate(((0, 1), (1, 2), (2, 0))):
        xa, ya = mesh.vx[mesh.etov[:, i]], mesh.vy[mesh.etov[:, i]]
        xb, yb = mesh.vx[mesh.etov[:, j]], mesh.vy[mesh.etov[:, j]]
        mesh.face_tag[:, f] = np.select([(ya == 0) & (yb == 0), (xa == 2) & (xb == 2), (ya == 1) & (yb == 1),
                                         (xa == 0) & (xb == 0)], [1, 2, 3, 4], 0)
    return mesh


def initial_state(problem, x, y, seed):
    """A smooth state [K][Np][m] at the node coordinates (device tensors), its
    strength, place and superposed waves drawn from the seed."""
    r = np.random.default_rng(seed)
    pi = math.pi
    if problem == "advection":
        u = 0.1 * torch.sin(2 * pi * (r.integers(1, 4) * x + r.integers(1, 4) * y) + r.uniform(0, 6))
        x0, y0, w = r.uniform(0.3, 0.7), r.uniform(0.3, 0.7), r.uniform(0.008, 0.02)
        return (u + torch.exp(-((x - x0) ** 2 + (y - y0) ** 2) / w))[..., None].contiguous()
    if problem == "vortex":
        beta, x0, y0 = r.uniform(1.0, 5.0), r.uniform(4.0, 6.0), r.uniform(4.0, 6.0)
        r2 = (x - x0) ** 2 + (y - y0) ** 2
        u = 1.0 - beta * torch.exp(1.0 - r2) * (y - y0) / (2 * pi)
        v = beta * torch.exp(1.0 - r2) * (x - x0) / (2 * pi)
        rho = (1.0 - 0.4 * beta * beta * torch.exp(2.0 * (1.0 - r2)) / (22.4 * pi * pi)) ** 2.5
        p = rho ** 1.4
        for f in range(1, 4):
            rho = rho * (1.0 + 0.01 * torch.sin(0.2 * pi * f * (x + y) + r.uniform(0, 6)))
            v = v + 0.02 * torch.cos(0.2 * pi * f * x + r.uniform(0, 6))
        return torch.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], dim=-1).contiguous()
    if problem == "channel":
        x0, a = r.uniform(0.7, 1.3), r.uniform(0.1, 0.3)
        rho = 1.0 + a * torch.exp(-((x - x0) ** 2 + (y - 0.5) ** 2) / 0.05)
        u, v = 0.5 + 0.05 * torch.sin(pi * y + r.uniform(0, 6)), 0.2 * torch.sin(pi * x + r.uniform(0, 6))
        w, p = 0.1 * torch.cos(pi * (x - y)), 1.0 + 0.3 * torch.cos(2 * pi * y + r.uniform(0, 6))
        return torch.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)],
                           dim=-1).contiguous()
    if problem == "cavity":
        ez, bx, by = 0.0, 0.0, 0.0
        for k in range(1, 4):
            a, ph, w = r.uniform(0.3, 1.0), r.uniform(0, 6), math.hypot(k, 1) * pi
            ez = ez + a * math.cos(ph) * torch.sin(k * pi * x) * torch.sin(pi * y)
            bx = bx - a * math.sin(ph) * pi / w * torch.sin(k * pi * x) * torch.cos(pi * y)
            by = by + a * math.sin(ph) * k * pi / w * torch.cos(k * pi * x) * torch.sin(pi * y)
        return torch.stack([ez, bx, by], dim=-1).contiguous()
    out = []
    for f in range(8):
        k, l, ph, a = r.integers(1, 4), r.integers(1, 4), r.uniform(0, 6), r.uniform(0.2, 1.0)
        out.append(a * torch.sin(int(k) * pi * x + ph) * torch.cos(int(l) * pi * y + ph))
    return torch.stack(out, dim=-1).contiguous()


def instances(case):
    """(order, vertex grid, mesh seed) of each instance of an ensemble."""
    got = []
    for i in range(case["count"]):
        k = case["kmin"] * (case["kmax"] / case["kmin"]) ** (i / max(1, case["count"] - 1))
        got.append((2 + i % 4, max(3, int(round(math.sqrt(k / 2)))) + 1, i))
    return got


def device_coords(xy):
    return [torch.from_numpy(a).cuda() for a in xy]


# ------------------------------------------------------------- the calls ----
def prepare(case, seed):
    p = case["problem"]
    kind, params, bcs, sources, flux = equation(p)
    if case["kind"] == "ensemble":
        b = NodalDG2dBatch(CFL, kind, params, bcs=bcs)
        for N, n, ms in instances(case):
            b.add_mesh(N, mesh_of(p, n, ms))
        b.finalize()
        U = [initial_state(p, *device_coords(b.node_coords(i)), seed=seed * 100 + i) for i in range(len(b))]
        for i, u in enumerate(U):
            b.set_state(i, u)
        return dict(case=case, batch=b, U=U, out=[torch.empty_like(u) for u in U], dt=b.init_dt())
    s = NodalDG2d(case["N"], CFL, kind, params, mesh_of(p, case["n"]), bcs=bcs, sources=sources, numerical_flux=flux)
    if case.get("limiter"):
        s.set_limiter("eulerLimiterHW", (1.4, 1e-4, 1e-4))
    x, y = device_coords(s.node_coords())
    U = initial_state(p, x, y, seed)
    s.set_state(U)
    st = dict(case=case, solver=s, U=U, out=torch.empty_like(U), dt=s.init_dt())
    if case["kind"] == "gradient":
        st["target"] = initial_state(p, x, y, seed + 50)
        st["grad"] = torch.empty_like(U)
    if case["kind"] == "jacobian":
        st["v"], st["w"] = direction(U, seed, 1), direction(U, seed, 2)
        st["vjp"] = torch.empty_like(U)
    return st


def direction(U, seed, which):
    """A seeded vector of the state's shape."""
    r = np.random.default_rng([seed, which])
    return torch.from_numpy(r.standard_normal(tuple(U.shape))).to(U.device)


def run(state):
    case, U, out = state["case"], state["U"], state["out"]
    if case["kind"] == "ensemble":
        b = state["batch"]
        for i, u in enumerate(U):
            b.set_state(i, u)
        t, dt = b.step(1, np.zeros(len(U)), state["dt"], precision=case["precision"])
        for i, o in enumerate(out):
            b.get_state(i, o)
        return {"U": out, "t": t, "dt": dt}
    s = state["solver"]
    if case["kind"] == "rhs":
        _, dt = s.step(0.0, state["dt"], U, out, precision=case["precision"])
        return {"rhs": out, "dt": dt}
    if case["kind"] == "jacobian":
        s.rhs_jvp(0.0, U, state["v"], out)
        s.rhs_vjp(0.0, U, state["w"], state["vjp"])
        return {"jvp": out, "vjp": state["vjp"]}
    s.set_state(U)
    if case["kind"] == "gradient":
        s.forward_fixed(case["steps"], 0.0, state["dt"], case["every"])
        s.get_state(out)
        s.backward(out - state["target"], out=state["grad"])
        return {"U": out, "grad": state["grad"]}
    t, dt = s.advance(case["steps"], 0.0, state["dt"], precision=case["precision"])
    s.get_state(out)
    return {"U": out, "t": t, "dt": dt}


NC = {2: 19, 3: 36, 4: 54, 5: 73}  # cubature points of an element by order


def work(case):
    """Per stage: the stage input read and its result written (and the step's
    start state in the last of five), the element geometry, and the multiply-adds
    of the element operators with their values used once."""
    if case["kind"] == "ensemble":
        parts = [work(dict(kind="step", problem=case["problem"], N=N, n=n, steps=1)) for N, n, _ in instances(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    N, m, K = case["N"], FIELDS[case["problem"]], 2 * (case["n"] - 1) ** 2
    Np, Nf, Nc = (N + 1) * (N + 2) // 2, 6 * (N + 1), NC[N]
    state, rhs = 8.0 * Np * m, 2.0 * m * (3 * Nc * Np + 2 * Nf * Np)
    if case["kind"] == "rhs":
        return {"bytes": K * (2 * state + 160), "flops": K * rhs}
    if case["kind"] == "jacobian":  # each way: the state and a vector in, a vector out
        return {"bytes": K * 2 * (3 * state + 160), "flops": K * 4 * rhs}
    stages = 5 * case["steps"]
    one = {"bytes": K * (stages * (2 * state + 160) + case["steps"] * state), "flops": K * stages * rhs}
    if case["kind"] == "gradient":  # forward, and per stage backwards its state and adjoint in, the adjoint out
        return {"bytes": one["bytes"] + K * stages * (3 * state + 160), "flops": 3 * one["flops"]}
    return one


# ------------------------------------------- the same in plain 64-bit torch ----
@functools.lru_cache(maxsize=None)
def tables(N):
    """Node set and cubature rule of order N (the discretisation's published
    numbers, read as data)."""
    here = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with open(os.path.join(here, "apollo_b200", "csrc", "dg_tables.inc")) as f:
        text = f.read()

    def numbers(name):
        return np.array([float(v) for v in re.search(name + r"_N%d\[\d+\] = \{(.*?)\}" % N, text, re.S)[1].split(",")
                         if v.strip()])

    return numbers("kNodeR"), numbers("kNodeS"), numbers("kCubRST").reshape(-1, 3)


def operators(N):
    """Nodal interpolation and weak-derivative matrices of order N."""
    r, s, cub = tables(N)
    powers = [(i, j) for i in range(N + 1) for j in range(N + 1 - i)]

    def mono(a, b, da=0, db=0):
        cols = []
        for i, j in powers:
            ca, cb = (i if da else 1), (j if db else 1)
            cols.append(ca * cb * a ** max(i - da, 0) * b ** max(j - db, 0))
        return np.stack(cols, axis=1)

    inv = np.linalg.inv(mono(r, s))
    z, gw = np.polynomial.legendre.leggauss(2 * (N + 1))
    one = np.ones_like(z)
    fr, fs = np.concatenate([z, -z, -one]), np.concatenate([-one, z, -z])
    cr, cs, w = cub.T
    V, I = mono(cr, cs) @ inv, mono(fr, fs) @ inv
    minv = np.linalg.inv(V.T @ (w[:, None] * V))
    Dr, Ds = (minv @ ((mono(cr, cs, *d) @ inv) * w[:, None]).T for d in ((1, 0), (0, 1)))
    return dict(r=r, s=s, cr=cr, cs=cs, V=V, I=I, Dr=Dr, Ds=Ds, S=minv @ (V * w[:, None]).T, L=minv @ I.T, z=z, gw=gw,
                fr=fr, fs=fs, rmin=abs(r[1] - r[0]))


class Plain:
    """The right-hand side and the stepper of one problem on one mesh."""

    def __init__(self, problem, N, mesh, device):
        self.problem, self.N = problem, N
        o = operators(N)
        self.ng = len(o["z"])
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)  # noqa: E731
        self.op = {k: to(o[k]) for k in ("V", "I", "Dr", "Ds", "S", "L", "gw")}
        ev = mesh.etov.astype(np.int64)
        vx, vy = mesh.vx[ev], mesh.vy[ev]
        at = lambda v, r, s: 0.5 * (-v[:, :1] * (r + s) + v[:, 1:2] * (1 + r) + v[:, 2:] * (1 + s))  # noqa: E731
        self.x, self.y = to(at(vx, o["r"], o["s"])), to(at(vy, o["r"], o["s"]))
        self.cx, self.cy = to(at(vx, o["cr"], o["cs"])), to(at(vy, o["cr"], o["cs"]))
        xr, xs, yr, ys = ((v[:, i] - v[:, 0]) / 2 for v in (vx, vy) for i in (1, 2))
        J = xr * ys - xs * yr
        self.rx, self.ry, self.sx, self.sy = (to(a / J)[:, None, None] for a in (ys, -xs, -yr, xr))
        self.iJ = to(1 / J)[:, None, None]
        ex, ey = np.roll(vx, -1, 1) - vx, np.roll(vy, -1, 1) - vy
        ln = np.hypot(ex, ey)
        wide = lambda a: to(np.repeat(a, self.ng, axis=1))  # noqa: E731
        self.nx, self.ny = wide(ey / ln), wide(-ex / ln)
        self.wf = wide(ln / 2) * self.op["gw"].repeat(3)
        sp = ln.sum(1) / 2
        area = np.sqrt(np.abs(sp * (sp - ln[:, 0]) * (sp - ln[:, 1]) * (sp - ln[:, 2])))
        self.dtfac = 2 / 3 * CFL * (area / sp).min() * o["rmin"]
        # the flat index of every face point's partner (its own where the face is a boundary)
        canon = mesh.vert_canon.astype(np.int64)[ev]
        a, b = canon, np.roll(canon, -1, 1)
        key = (np.minimum(a, b) * (canon.max() + 1) + np.maximum(a, b)).ravel()
        tag = mesh.face_tag.ravel()
        order = np.argsort(key, kind="stable")
        partner = np.full(key.size, -1)
        same = np.flatnonzero(key[order][1:] == key[order][:-1])
        partner[order[same]], partner[order[same + 1]] = order[same + 1], order[same]
        partner[tag > 0] = -1
        own = np.arange(key.size)[:, None] * self.ng + np.arange(self.ng)
        other = partner[:, None] * self.ng + np.arange(self.ng)[::-1]
        self.other = to(np.where(partner[:, None] >= 0, other, own).ravel())
        self.tag = to(np.repeat(np.where(partner >= 0, 0, np.maximum(tag, 1)), self.ng).reshape(len(ev), -1))

    def flux(self, q):
        """(F, G) of states [..., m]."""
        p = self.problem
        if p == "advection":
            return q, 0.5 * q
        if p == "cavity":
            z = torch.zeros_like(q[..., 0])
            return torch.stack([-q[..., 2], z, -q[..., 0]], -1), torch.stack([q[..., 1], q[..., 0], z], -1)
        if p == "cleaning":
            ex, ey, ez, bx, by, bz, ph, ps = q.unbind(-1)
            g, c = 0.8, 0.6
            return (torch.stack([c * ph, bz, -by, g * ps, -ez, ey, c * ex, g * bx], -1),
                    torch.stack([-bz, c * ph, bx, ez, g * ps, -ex, c * ey, g * by], -1))
        rho, E = q[..., 0], q[..., -1]
        vel = [q[..., i] / rho for i in range(1, q.shape[-1] - 1)]
        pr = 0.4 * (E - 0.5 * rho * sum(v * v for v in vel))
        out = []
        for d in (0, 1):
            f = [rho * vel[d]] + [rho * v * vel[d] for v in vel] + [(E + pr) * vel[d]]
            f[1 + d] = f[1 + d] + pr
            out.append(torch.stack(f, -1))
        return out

    def primitive(self, q):
        rho = q[..., 0]
        vel = [q[..., i] / rho for i in range(1, q.shape[-1] - 1)]
        return rho, vel, 0.4 * (q[..., -1] - 0.5 * rho * sum(v * v for v in vel))

    def speed(self, qM, qP):
        if self.problem in ("advection", "cavity", "cleaning"):
            return torch.ones_like(qM[..., 0])
        c = []
        for q in (qM, qP):
            rho, vel, p = self.primitive(q)
            c.append(torch.sqrt(sum(v * v for v in vel)) + torch.sqrt(1.4 * p / rho))
        return torch.maximum(*c)

    def boundary(self, q):
        """The states outside the boundary faces [K, Nf, m]."""
        p, nx, ny = self.problem, self.nx, self.ny
        f = list(q.unbind(-1))
        if p == "cavity":
            return torch.stack([-f[0], f[1], f[2]], -1)
        if p == "cleaning":
            en, et = f[0] * nx + f[1] * ny, f[0] * ny - f[1] * nx
            bn, bt = -f[3] * nx - f[4] * ny, -f[3] * ny + f[4] * nx
            return torch.stack([en * nx - et * ny, en * ny + et * nx, -f[2], bn * nx - bt * ny, bn * ny + bt * nx, f[5],
                                -f[6], f[7]], -1)
        if p != "channel":
            return q
        mn = f[1] * nx + f[2] * ny
        wall = torch.stack([f[0], f[1] - 2 * mn * nx, f[2] - 2 * mn * ny, 0 * f[3], f[4]], -1)
        mach, angle, gamma, pr, rho = INFLOW
        c = mach * math.sqrt(gamma * pr / rho)
        u, v = c * math.cos(math.radians(angle)), c * math.sin(math.radians(angle))
        inflow = q.new_tensor([rho, rho * u, rho * v, 0.0, pr / (gamma - 1) + 0.5 * rho * (u * u + v * v)])
        rho, u, v, w, gamma, pr = DIRICHLET
        fixed = q.new_tensor([rho, rho * u, rho * v, rho * w, pr / (gamma - 1) + 0.5 * rho * (u * u + v * v + w * w)])
        tag = self.tag[..., None]
        return torch.where(tag == 1, wall, torch.where(tag == 3, inflow, torch.where(tag == 4, fixed, q)))

    def hll(self, qM, qP):
        """Apollo's HLL flux, whose bound |S_R| is truncated to a whole number."""
        nx, ny = self.nx, self.ny

        def turned(q):
            f = list(q.unbind(-1))
            return torch.stack([f[0], nx * f[1] + ny * f[2], -ny * f[1] + nx * f[2]] + f[3:], -1)

        a, b = turned(qM), turned(qP)
        fa, fb = self.flux(a)[0], self.flux(b)[0]
        (ra, va, pa), (rb, vb, pb) = self.primitive(a), self.primitive(b)
        wa, wb = torch.sqrt(ra), torch.sqrt(rb)
        mean = lambda x, y: (wa * x + wb * y) / (wa + wb)  # noqa: E731
        vel = [mean(x, y) for x, y in zip(va, vb)]
        H = mean((a[..., -1] + pa) / ra, (b[..., -1] + pb) / rb)
        c = torch.sqrt(0.4 * (H - 0.5 * sum(v * v for v in vel)))
        SL = torch.minimum(va[0] - torch.sqrt(1.4 * pa / ra), vel[0] - c)
        SR = torch.maximum(vb[0] + torch.sqrt(1.4 * pb / rb), vel[0] + c)
        t1 = (SR.clamp(max=0) - SL.clamp(max=0)) / (SR - SL)
        t3 = (SR * SL.abs() - SL * SR.trunc().abs()) / (2 * (SR - SL))
        fx = t1[..., None] * fb + (1 - t1)[..., None] * fa - t3[..., None] * (b - a)
        g = list(fx.unbind(-1))
        return torch.stack([g[0], nx * g[1] - ny * g[2], ny * g[1] + nx * g[2], 0 * g[0], g[-1]], -1)

    def rhs(self, u, t):
        """(L(u), the largest numerical-flux speed)."""
        o = self.op
        F, G = self.flux(torch.matmul(o["V"], u))
        out = torch.matmul(o["Dr"], self.rx * F + self.ry * G) + torch.matmul(o["Ds"], self.sx * F + self.sy * G)
        if self.problem == "cleaning":
            x, y = self.cx, self.cy
            src = math.exp(t) * (x * (1 - x) * y * (1 - y) + 2 * x * (1 - x) + 2 * y * (1 - y))
            pad = torch.zeros_like(out)
            pad[..., 2] = torch.matmul(o["S"], src[..., None])[..., 0]
            out = out + pad
        qM = torch.matmul(o["I"], u)
        qP = qM.reshape(-1, u.shape[-1])[self.other].reshape(qM.shape)
        if (self.tag > 0).any():
            qP = torch.where((self.tag > 0)[..., None], self.boundary(qM), qP)
        lam = self.speed(qM, qP)
        if self.problem == "channel":
            f = self.hll(qM, qP)
        else:
            (FM, GM), (FP, GP) = self.flux(qM), self.flux(qP)
            f = 0.5 * (self.nx[..., None] * (FM + FP) + self.ny[..., None] * (GM + GP) + lam[..., None] * (qM - qP))
        return out - self.iJ * torch.matmul(o["L"], self.wf[..., None] * f), lam

    def step(self, u, t, dt):
        w, lam = u, None
        for i in range(4):
            w = w + dt / 4 * self.rhs(w, t + dt * i / 4)[0]
        L, lam = self.rhs(w, t + dt)
        return 0.8 * w + dt / 5 * L + 0.2 * u, lam

    def first_dt(self, u):
        if self.problem in ("advection", "cavity", "cleaning"):
            return self.dtfac
        rho, vel, p = self.primitive(u)
        c = torch.maximum(vel[0].abs(), vel[1].abs()) + torch.sqrt(1.4 * p / rho)
        return self.dtfac / float(c.max())

    def advance(self, u, steps):
        t, dt = 0.0, self.first_dt(u)
        for _ in range(steps):
            u, lam = self.step(u, t, dt)
            t, dt = t + dt, min(dt, self.dtfac / float(lam.max()))
        return u, t, dt


def exact(case, seed):
    if case.get("limiter"):
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    p = case["problem"]
    if case["kind"] == "ensemble":
        got = []
        for i, (N, n, ms) in enumerate(instances(case)):
            d = Plain(p, N, mesh_of(p, n, ms), device)
            got.append(d.advance(initial_state(p, d.x, d.y, seed * 100 + i), 1))
        return {"U": [g[0] for g in got], "t": np.array([g[1] for g in got]), "dt": np.array([g[2] for g in got])}
    d = Plain(p, case["N"], mesh_of(p, case["n"]), device)
    U = initial_state(p, d.x, d.y, seed)
    if case["kind"] == "rhs":
        L, lam = d.rhs(U, 0.0)
        return {"rhs": L, "dt": d.dtfac / float(lam.max())}
    if case["kind"] == "jacobian":
        f = lambda u: d.rhs(u, 0.0)[0]  # noqa: E731
        with torch.enable_grad():
            leaf = U.clone().requires_grad_(True)
            L = f(leaf)
            (vjp,) = torch.autograd.grad(L, leaf, direction(U, seed, 2), create_graph=False)
            # the tangent as the derivative of the adjoint along its argument
            w = torch.zeros_like(U, requires_grad=True)
            (g,) = torch.autograd.grad(f(leaf), leaf, w, create_graph=True)
            (jvp,) = torch.autograd.grad(g, w, direction(U, seed, 1))
        return {"jvp": jvp, "vjp": vjp}
    if case["kind"] == "gradient":
        dt = d.first_dt(U)
        with torch.enable_grad():
            leaf = U.clone().requires_grad_(True)
            u = leaf
            for k in range(case["steps"]):
                u = torch.utils.checkpoint.checkpoint(lambda v, k=k: d.step(v, k * dt, dt)[0], u, use_reentrant=False)
            end = u.detach()
            (grad,) = torch.autograd.grad(u, leaf, end - initial_state(p, d.x, d.y, seed + 50))
        return {"U": end, "grad": grad}
    u, t, dt = d.advance(U, case["steps"])
    return {"U": u, "t": t, "dt": dt}
