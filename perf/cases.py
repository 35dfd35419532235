"""Workloads of the framework, as a program that uses it calls them: what is timed
and compared when a kernel changes.

A pass of every stepping case is a short solve through the public entry points:
the initial state goes in from device memory (kg_set_state_device), the solve
advances by a number of steps, and the state comes back into device memory in
the same layout (kg_get_state_device).  The kinds, and what each stands for:

* ``evolve``   -- the reference's evolve loop: single PIRK2 steps, each followed
  by the density and the mass integral, whose value the host reads.
* ``steps``    -- many steps of one stepper per call (pirk2, pirk3, rk3, rk4),
  FP64 or mixed precision (rk4), with the detector diagnostics at the end.
* ``batch``    -- one quantum of the continuous-batching server: ragged solves
  advanced together by RK4, then every solve's detector a_lm.
* ``refine``   -- radially nested 2:1 levels advanced together.
* ``config``   -- the fourth-order method with dissipation.
* ``spectral`` -- the Y_lm projection over every shell, and the spherical-Bessel
  transform on top of it, returned to the host.

`exact` restates the same mathematics in plain torch, in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from kg_b200 import ScalarField
from kg_b200.batch import Batch
from kg_b200.refinement import BergerOliger

DEV = "cuda:0"
G = 2  # ghost points per side


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest grid of the tests, stepped the way main/evolve.f90 steps: one
        # call per step, one number read per step -- launches and latency count
        dict(name="evolve-64x17x33", kind="evolve", Nx=64, Ny=17, Nz=33, steps=40, metric="Kerr_Schild",
             bc="outflow", m=0.3),
        # the reference's default grid, steps handed over in one call
        dict(name="pirk2-256x33x65", kind="steps", stepper="pirk2", Nx=256, Ny=33, Nz=65, steps=60,
             metric="Kerr_Schild", bc="outflow", m=0.0),
        # the large solve of the benchmark
        dict(name="pirk2-2048x129x257", kind="steps", stepper="pirk2", Nx=2048, Ny=129, Nz=257, steps=10,
             metric="Kerr_Schild", bc="outflow", m=0.3),
        # a ragged grid, with the other metric and the other outer boundary
        dict(name="rk4-301x46x90", kind="steps", stepper="rk4", Nx=301, Ny=46, Nz=90, steps=20, metric="Schw_EF",
             bc="inflow", m=0.2),
        # a radial grid of the batched benchmark's upper range, FP64 and mixed
        dict(name="rk4-1024x65x129", kind="steps", stepper="rk4", Nx=1024, Ny=65, Nz=129, steps=10,
             metric="Kerr_Schild", bc="outflow", m=0.3),
        dict(name="rk4mixed-1024x65x129", kind="steps", stepper="rk4mixed", Nx=1024, Ny=65, Nz=129, steps=10,
             metric="Kerr_Schild", bc="outflow", m=0.3),
        # the third-order PIRK method on a middle-sized grid
        dict(name="pirk3-512x65x129", kind="steps", stepper="pirk3", Nx=512, Ny=65, Nz=129, steps=10,
             metric="Kerr_Schild", bc="outflow", m=0.1),
        # a serving quantum: Nr 128..512, Ntheta 16 or 32, ten RK4 steps
        dict(name="batch-mixed-16", kind="batch", count=16, nr_max=512, precision="mixed", dispatch=0, steps=10),
        dict(name="batch-fp64-12", kind="batch", count=12, nr_max=512, precision="fp64", dispatch=1, steps=10),
        # two refined levels around the hole
        dict(name="refine-512x33x65", kind="refine", stepper="rk4", Nx=512, Ny=33, Nz=65, levels=3, steps=4),
        # the configured method on the grid its description names
        dict(name="config-256x33x65", kind="config", Nx=256, Ny=33, Nz=65, steps=20),
        # waveform extraction on every shell by the tensor-core projection
        dict(name="spectral-512x65x129-l32", kind="spectral", Nx=512, Ny=65, Nz=129, L=32, precision=1, Nk=0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evolve", "steps", "steps", "steps", "batch", "refine", "config", "spectral"])
    metric = rng.choice(["Kerr_Schild", "Kerr_Schild", "Schw_EF"])
    bc = rng.choice(["outflow", "outflow", "inflow"])
    m = round(rng.uniform(0.0, 0.5), 3)
    if kind == "evolve":
        return dict(kind=kind, Nx=_logint(rng, 24, 400), Ny=_logint(rng, 9, 49), Nz=_logint(rng, 17, 97),
                    steps=rng.randint(5, 40), metric=metric, bc=bc, m=m)
    if kind == "steps":
        stepper = rng.choice(["pirk2", "pirk2", "pirk3", "rk3", "rk4", "rk4mixed"])
        while True:
            c = dict(kind=kind, stepper=stepper, Nx=_logint(rng, 32, 2048), Ny=_logint(rng, 9, 129),
                     Nz=_logint(rng, 17, 257), steps=rng.randint(2, 20), metric=metric, bc=bc, m=m)
            stages = {"pirk2": 2, "pirk3": 3, "rk3": 3}.get(stepper, 4)
            if _stored(c) * c["steps"] * stages <= 7.0e8:  # half of the largest listed case
                return c
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), nr_max=128 * rng.randint(1, 4),
                    precision=rng.choice(["fp64", "mixed"]), dispatch=rng.choice([0, 1]), steps=rng.randint(2, 10))
    if kind == "refine":
        return dict(kind=kind, stepper=rng.choice(["rk4", "pirk2"]), Nx=_logint(rng, 96, 600),
                    Ny=_logint(rng, 9, 49), Nz=_logint(rng, 17, 97), levels=rng.randint(2, 3),
                    steps=rng.randint(1, 4))
    if kind == "config":
        return dict(kind=kind, Nx=_logint(rng, 32, 512), Ny=_logint(rng, 9, 65), Nz=_logint(rng, 17, 129),
                    steps=rng.randint(2, 12))
    return dict(kind=kind, Nx=_logint(rng, 32, 800), Ny=_logint(rng, 17, 97), Nz=_logint(rng, 33, 193),
                L=rng.randint(4, 40), precision=rng.choice([0, 1]), Nk=rng.choice([0, 0, rng.randint(4, 24)]))


def _stored(c):
    return (c["Nx"] + 5) * (c["Ny"] + 5) * (c["Nz"] + 1)


def _domain(Nx):
    """r in [1.8, xmax]: the benchmark's spacing, on at least the first 12 radii"""
    return 1.8, 1.8 + max(12.0, 398.2 * Nx / 2048)


def _members(c, seed):
    """the grids of a batch: Nr in steps of 64 up to nr_max, Ntheta 16 or 32, Nphi twice that"""
    r = np.random.default_rng(9000 + 7 * c["count"] + c["nr_max"])  # the shapes belong to the case
    out = []
    for i in range(c["count"]):
        nt = int(r.choice([16, 32]))
        nx = int(r.choice(np.arange(128, c["nr_max"] + 1, 64)))
        out.append(dict(Nx=nx, Ny=nt + 1, Nz=2 * nt + 1, metric="Kerr_Schild", bc="outflow",
                        m=float(np.round(r.uniform(0.0, 0.5), 3)), seed=seed * 1000 + i))
    return out


def _radii(c):
    """outer radii of the refined levels"""
    x0, x1 = _domain(c["Nx"])
    return tuple(x0 + (x1 - x0) * f for f in (0.4, 0.15)[: c["levels"] - 1])


# ---------------------------------------------------------------------------
# initial data: a Gaussian shell times a random polynomial of degree 4 in the
# direction (l <= 4), psi_i from the reference's second-order stencils, Pi = 0

def _axes(Nx, Ny, Nz, xmin, xmax):
    dx, dy, dz = (xmax - xmin) / Nx, math.pi / (Ny - 1), 2.0 * math.pi / (Nz - 1)
    x = xmin + torch.arange(Nx + 5, dtype=torch.float64, device=DEV) * dx
    y = -dy / 2.0 + torch.arange(-G, Ny + G + 1, dtype=torch.float64, device=DEV) * dy
    z = torch.arange(Nz + 1, dtype=torch.float64, device=DEV) * dz
    return x, y, z, dx, dy, dz


def _d_r(f, h):
    d = torch.empty_like(f)
    d[..., 1:-1] = f[..., 2:] - f[..., :-2]
    d[..., 0] = -3.0 * f[..., 0] + 4.0 * f[..., 1] - f[..., 2]
    d[..., -1] = 3.0 * f[..., -1] - 4.0 * f[..., -2] + f[..., -3]
    return d.mul_(0.5 / h)


def _partner(NK):
    Nz = NK - 1
    return [(k + Nz // 2) % (Nz - 1) for k in range(NK)]


def _d_th(f, h):
    d = torch.empty_like(f)
    d[:, 1:-1] = f[:, 2:] - f[:, :-2]
    d[:, 0] = f[_partner(f.shape[0]), 2] - f[:, 1]
    d[:, -1] = 3.0 * f[:, -1] - 4.0 * f[:, -2] + f[:, -3]
    return d.mul_(0.5 / h)


def _d_ph(f, h):
    d = torch.empty_like(f)
    n = f.shape[0] - 1
    d[1:-1] = f[2:] - f[:-2]
    d[0] = f[1] - f[n - 2]
    d[n] = f[n - 1] - f[2]
    return d.mul_(0.5 / h)


def _initial(Nx, Ny, Nz, xmin, xmax, seed):
    r = np.random.default_rng(seed)
    r0, sd = float(r.uniform(5.0, 9.0)), float(r.uniform(1.0, 2.0))
    poly = [complex(*r.normal(size=2))] + [(complex(*r.normal(size=2)), r.normal(size=3)) for _ in range(8)]
    x, y, z, dx, dy, dz = _axes(Nx, Ny, Nz, xmin, xmax)
    s, c = torch.sin(y)[None, :], torch.cos(y)[None, :]
    n = (s * torch.cos(z)[:, None], s * torch.sin(z)[:, None], c.expand(Nz + 1, -1))
    ang = torch.full((Nz + 1, Ny + 5), poly[0], dtype=torch.complex128, device=DEV)
    for i, (a, v) in enumerate(poly[1:]):
        v = v / np.linalg.norm(v)
        ang += a * (float(v[0]) * n[0] + float(v[1]) * n[1] + float(v[2]) * n[2]) ** (1 + i // 2)
    phi = ang[:, :, None] * torch.exp(-((x - r0) / sd) ** 2)[None, None, :]
    u = torch.empty((Nz + 1, Ny + 5, Nx + 5, 5), dtype=torch.complex128, device=DEV)
    u[..., 0] = phi
    u[..., 1] = _d_r(phi, dx)
    u[..., 2] = _d_th(phi, dy)
    u[..., 3] = _d_ph(phi, dz)
    u[..., 4] = 0.0
    return u


# ---------------------------------------------------------------------------
# preparing and running

class _Solve:
    """a solver with its initial state and the buffer its result goes to"""

    def __init__(self, s, u0):
        self.s, self.u0, self.out = s, u0, torch.empty_like(u0)

    def put(self):
        s = self.s
        s._ck(s._lib.kg_set_state_device(s.handle, 0, C.c_void_p(self.u0.data_ptr())))

    def get(self):
        s = self.s
        s._ck(s._lib.kg_get_state_device(s.handle, 0, C.c_void_p(self.out.data_ptr())))
        return self.out


def _solve(c, seed):
    x0, x1 = _domain(c["Nx"])
    s = ScalarField(c["Nx"], c["Ny"], c["Nz"], x0, x1, 0.25, m=c.get("m", 0.3),
                    metric=c.get("metric", "Kerr_Schild"), boundary_type_rmax=c.get("bc", "outflow"), l_max=8)
    return _Solve(s, _initial(c["Nx"], c["Ny"], c["Nz"], x0, x1, seed))


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        st = dict(case=c, solves=[_solve(g, g["seed"]) for g in _members(c, seed)],
                  batch=Batch(precision=c["precision"]))
        for v in st["solves"]:
            st["batch"].add(v.s)
        st["batch"].set_tuning(32, 296, dispatch=c["dispatch"])
    elif c["kind"] == "refine":
        x0, x1 = _domain(c["Nx"])
        bo = BergerOliger(c["Nx"], c["Ny"], c["Nz"], x0, x1, 0.25, r_fine=_radii(c), m=0.3, l_max=8)
        st = dict(case=c, bo=bo, solves=[
            _Solve(lv, _initial(lv.Nx, lv.Ny, lv.Nz, x0, float(lv.params.xmax), seed)) for lv in bo.levels])
    else:
        st = dict(case=c, solves=[_solve(c, seed)])
        s = st["solves"][0].s
        if c.get("stepper") == "rk4mixed":
            s.precision = "mixed"
        if c["kind"] == "config":
            s.set_scheme("configured")
        if c["kind"] == "spectral":  # the state a projection reads is there already
            st["solves"][0].put()
            s.synchronize()
    torch.cuda.synchronize()  # the solver reads the inputs on its own stream
    return st


def run(state):
    c = state["case"]
    solves = state["solves"]
    s = solves[0].s
    if c["kind"] == "spectral":
        if c["Nk"]:
            return s.sph_ft_radial(c["L"], c["Nk"], precision=c["precision"])
        return s.project_all_shells(c["L"], precision=c["precision"])
    for v in solves:
        v.put()
    if c["kind"] == "evolve":
        mass = []
        for step in range(1, c["steps"] + 1):
            s.pirk2()
            s.density()
            mass.append(s.diagnostic(step))
        return [solves[0].get(), np.array(mass)]
    if c["kind"] == "batch":
        state["batch"].rk4(c["steps"])
        alm = state["batch"].proyector_detectors()
        return [[v.get() for v in solves], alm]
    if c["kind"] == "refine":
        getattr(state["bo"], c["stepper"])(c["steps"])
        return [v.get() for v in solves]
    if c["kind"] == "config":
        s.fill_ghosts_configured()
        s.rk4(nsteps=c["steps"])
        return solves[0].get()
    getattr(s, c["stepper"].replace("mixed", ""))(nsteps=c["steps"])
    s.density()
    mass = s.mass_scalar()
    momentum = s.currents_detectors().copy()
    alm = s.proyector_detectors().copy()
    return [solves[0].get(), mass, momentum, alm]


def work(case):
    """Bytes: the initial state in and the result out (80 B per stored point each),
    and per step the state read and written once (160 B; the stage sums of a step
    need not leave the chip), with the previous step's Pi of the PIRK methods
    (32 B); for the projection, phi in and the coefficients out.  Operations: the
    five right-hand sides and the stage update at every stored point, about 200 a
    stage (580 for the fourth-order method with dissipation); for the projection,
    the real products of its contraction."""
    c = case
    if c["kind"] == "spectral":
        sphere, modes = c["Ny"] * c["Nz"], (c["L"] + 1) * (c["L"] + 2) // 2
        out = 16 * c["Nx"] * (c["L"] + 1) * (2 * c["L"] + 1)
        flops = 2.0 * (2 * c["Nx"]) * sphere * (2 * modes)
        if c["Nk"]:
            flops += 4.0 * c["Nx"] * c["Nk"] * (c["L"] + 1) * (2 * c["L"] + 1)
            out = 16 * c["Nk"] * (c["L"] + 1) * (2 * c["L"] + 1)
        return {"bytes": 16.0 * c["Nx"] * sphere + out, "flops": flops}
    if c["kind"] == "batch":
        pts = [(_stored(g), 1) for g in _members(c, 0)]
    elif c["kind"] == "refine":
        x0, x1 = _domain(c["Nx"])
        dx = (x1 - x0) / c["Nx"]
        nx = [c["Nx"]] + [int((r - x0) / (dx / 2 ** (l + 1))) for l, r in enumerate(_radii(c))]
        pts = [(_stored(dict(c, Nx=n)), 2 ** l) for l, n in enumerate(nx)]
    else:
        pts = [(_stored(c), 1)]
    stepper = c.get("stepper", "pirk2" if c["kind"] == "evolve" else "rk4")
    per = 192.0 if stepper.startswith("pirk") else 160.0
    stages = {"pirk2": 2, "pirk3": 3, "rk3": 3}.get(stepper, 4)
    ops = 580.0 if c["kind"] == "config" else 200.0
    return {"bytes": sum(p * (160.0 + per * n * c["steps"]) for p, n in pts),
            "flops": sum(p * ops * stages * n * c["steps"] for p, n in pts)}


# ---------------------------------------------------------------------------
# the same mathematics in plain torch, 64 bits

class _Exact:
    """The method of lines on the whole grid, in array form (variables of shape
    (phi, theta, r)); metric_kind, boundaries and steppers as the solver's."""

    def __init__(self, Nx, Ny, Nz, xmin, xmax, m=0.3, metric="Kerr_Schild", bc="outflow", dt=None):
        self.Nx, self.Ny, self.Nz, self.NK = Nx, Ny, Nz, Nz + 1
        self.ks, self.inflow, self.m2 = metric == "Kerr_Schild", bc == "inflow", m * m
        self.xmin, self.xmax = xmin, xmax
        x, y, z, self.dx, self.dy, self.dz = _axes(Nx, Ny, Nz, xmin, xmax)
        self.x = x
        e = math.exp(xmin)
        self.dt = dt or 0.25 * min(self.dx, e * self.dy, e * math.sin(self.dy / 2.0) * self.dz)
        # M = 1, no spin: g_tt = -1 + 2/r, g_tr = 2/r, g_rr = 1 + 2/r, g_thth = r^2, g_phph = r^2 sin^2
        r = x[None, :].expand(len(y), -1)
        sn = torch.sin(y)[:, None].expand(-1, len(x)).clone()
        sn[-1] = sn[-2]  # the last theta row takes the metric of the row before it
        h = 2.0 / r
        self.al = 1.0 / torch.sqrt(1.0 + h)
        self.be = h / (1.0 + h)
        self.sg = r * r * torch.abs(sn) * torch.sqrt(1.0 + h)
        self.grr, self.gtt, self.gpp = 1.0 / (1.0 + h), 1.0 / (r * r), 1.0 / (r * r * sn * sn)
        self.dbe = _d_r(self.be, self.dx)
        self.S = self.T = None  # stage arrays: PIRK reads the previous step's Pi from them
        self.pos, self.neg = self.be > 0, self.be < 0

    def up_r(self, f):
        """first-order-accurate-at-the-ends upwind difference along r, by the sign of beta"""
        d = torch.empty_like(f)
        fw = -3.0 * f[..., :-2] + 4.0 * f[..., 1:-1] - f[..., 2:]
        d[..., :-2] = fw
        d[..., -1] = 3.0 * f[..., -1] - 4.0 * f[..., -2] + f[..., -3]
        d[..., -2] = f[..., -1] - f[..., -3]
        return d.mul_(0.5 / self.dx)  # beta > 0 everywhere outside and inside the horizon

    def rhs_psi(self, v):
        E = self.al * v[4] + self.be * v[1]
        r1 = _d_r(self.al * v[4], self.dx)
        r1 += self.be * self.up_r(v[1])
        r1 += self.dbe * v[1]
        return [E, r1, _d_th(E, self.dy), _d_ph(E, self.dz)]

    def rhs_pi(self, v):
        a = self.al * self.sg
        r = _d_r((a * self.grr) * v[1], self.dx)
        r += _d_th((a * self.gtt) * v[2], self.dy)
        r += _d_ph((a * self.gpp) * v[3], self.dz)
        r += self.be * self.up_r(self.sg * v[4])
        r /= self.sg
        r += self.dbe * v[4]
        r -= (self.al * self.m2) * v[0]
        return r

    def rhs(self, v):
        return self.rhs_psi(v) + [self.rhs_pi(v)]

    def fill(self, u, hold):
        for w in range(5):
            f = u[w]
            f[..., 0] = 3.0 * f[..., 1] - 3.0 * f[..., 2] + f[..., 3]
            f[..., -1] = hold[w][..., -1] if self.inflow else f[..., -2]
            self._poles(f, 1.0)
            f[0] = f[self.Nz - 1]
            f[self.Nz] = f[1]
        return u

    def _poles(self, f, sign):
        kt, n = _partner(self.NK), f.shape[1]
        for g in range(3):
            f[:, g] = sign * f[:, 5 - g][kt]
            f[:, n - 1 - g] = sign * f[:, n - 6 + g][kt]

    def pirk_1(self, u):
        dt = self.dt
        if self.S is None:
            self.S = [torch.zeros_like(f) for f in u]
        s = [f + dt * r for f, r in zip(u[:4], self.rhs_psi(u))]
        self.S = s + [u[4] + dt * self.rhs_pi(s + [self.S[4]])]
        return self.S

    def pirk2(self, u, between=None):
        s = self.pirk_1(u)
        if between:
            between(s, 1.0)
        n = []
        for f, g, r in zip(u, s, self.rhs(s)):
            n.append((f + g + self.dt * r).mul_(0.5))
        return self.fill(n, u)

    def pirk3(self, u):
        dt, s = self.dt, self.pirk_1(u)
        if self.T is None:
            self.T = [torch.zeros_like(f) for f in u]
        t = [0.75 * f + 0.25 * (g + dt * r) for f, g, r in zip(u[:4], s[:4], self.rhs_psi(s))]
        self.T = t + [0.75 * u[4] + 0.25 * (s[4] + dt * self.rhs_pi(t + [self.T[4]]))]
        n = [f / 3.0 + (g + dt * r) * (2.0 / 3.0) for f, g, r in zip(u, self.T, self.rhs(self.T))]
        return self.fill(n, u)

    def rk3(self, u):
        dt = self.dt
        a = self.fill([f + dt * r for f, r in zip(u, self.rhs(u))], u)
        b = self.fill([0.75 * f + 0.25 * (g + dt * r) for f, g, r in zip(u, a, self.rhs(a))], u)
        return self.fill([f / 3.0 + (g + dt * r) * (2.0 / 3.0) for f, g, r in zip(u, b, self.rhs(b))], u)

    def rk4(self, u, between=None, rhs=None, fill=None):
        dt, rhs, fill = self.dt, rhs or self.rhs, fill or self.fill
        acc, v = None, u
        for c, w, at in ((0.5, 1.0, 0.5), (0.5, 2.0, 0.5), (1.0, 2.0, 1.0), (None, 1.0, 1.0)):
            k = rhs(v)
            acc = [w * dt * r for r in k] if acc is None else [a + w * dt * r for a, r in zip(acc, k)]
            v = [f + c * dt * r for f, r in zip(u, k)] if c else [f + a / 6.0 for f, a in zip(u, acc)]
            fill(v, u)
            if between and c:
                between(v, at)
        return v

    rk4mixed = rk4

    # diagnostics (the detectors' radii, momenta and a_lm; the mass)
    def density(self, u):
        a = [torch.abs(f) for f in u]
        return 0.5 * (a[4] + self.grr * a[1] ** 2 + self.gtt * a[2] ** 2 + self.gpp * a[3] ** 2 + self.m2 * a[0])

    def mass(self, u):
        q = (self.density(u) * self.sg)[:, 2:-2, 2:-2]
        for d in range(3):
            n = q.shape[0]
            q = q.sum(0) - 0.5 * (q[0] + q[n - 1])  # phi, then theta, then r
        return float(q * self.dx * self.dy * self.dz)

    def detectors(self, n=5):
        r0, r1 = 2.0, 0.99 * self.xmax
        r = [r0] + [r0 + (r1 - r0) / n * (d - 1) for d in range(2, n)] + [r1]
        return [int((q - self.xmin) / self.dx) if self.xmin <= q < self.xmin + (self.Nx - 1) * self.dx else -1 for q in r]

    def shell(self, f, i):
        """a field at vertex radius i: the vertex rows lie midway between the stored theta rows"""
        q = f[: self.Nz, :, i]
        return 0.5 * (q[:, 2:2 + self.Ny] + q[:, 3:3 + self.Ny])

    def momentum(self, u, n=5):
        w = _trapezium(self.Nz)[:, None] * _trapezium(self.Ny)[None, :] * (self.dy * self.dz)
        out = np.zeros((n, 3))
        for d, i in enumerate(self.detectors(n)):
            if i < 0:
                continue
            for c, (g, f) in enumerate(((self.grr, u[1]), (self.gtt, u[2]), (self.gpp, u[3]))):
                j = -u[4][:, :, i] * f[:, :, i] * (g * self.sg)[:, i]
                q = 0.5 * (j[: self.Nz, 2:2 + self.Ny] + j[: self.Nz, 3:3 + self.Ny])
                out[d, c] = float((w * q).sum().real)
        return out

    def alm(self, shells, L):
        """a_lm of shells (n, Nz, Ny): (n, 2L+1, L+1)"""
        th = torch.arange(self.Ny, dtype=torch.float64, device=DEV) * self.dy
        ph = torch.arange(self.Nz, dtype=torch.float64, device=DEV) * self.dz
        w = _trapezium(self.Nz)[:, None] * (_trapezium(self.Ny) * torch.sin(th))[None, :] * (self.dy * self.dz)
        out = torch.zeros((shells.shape[0], 2 * L + 1, L + 1), dtype=torch.complex128, device=DEV)
        P = _legendre(L, th)
        q = shells * w
        for m in range(-L, L + 1):
            f = torch.einsum("nkj,k->nj", q, torch.exp(-1j * m * ph))
            a = torch.einsum("nj,lj->nl", f, P[:, abs(m)].to(torch.complex128))
            out[:, m + L] = a * ((-1.0) ** m if m < 0 else 1.0)
        return out

    def alm_detectors(self, u, L=8, n=5):
        out = np.zeros((n, 2 * L + 1, L + 1), np.complex128)
        for d, i in enumerate(self.detectors(n)):
            if i >= 0:
                out[d] = self.alm(self.shell(u[0], i)[None], L)[0].cpu().numpy()
        return out

    # the configured method: fourth-order differences, dissipation, Sommerfeld outer plane
    def d4_r(self, f):
        d = torch.empty_like(f)
        d[..., 2:-2] = f[..., :-4] - 8.0 * f[..., 1:-3] + 8.0 * f[..., 3:-1] - f[..., 4:]
        for o, s in ((0, 1.0), (-1, -1.0)):
            a = [f[..., i] if o == 0 else f[..., -1 - i] for i in range(5)]
            d[..., o] = s * (-25.0 * a[0] + 48.0 * a[1] - 36.0 * a[2] + 16.0 * a[3] - 3.0 * a[4])
            d[..., 1 if o == 0 else -2] = s * (-3.0 * a[0] - 10.0 * a[1] + 18.0 * a[2] - 6.0 * a[3] + a[4])
        return d.mul_(1.0 / (12.0 * self.dx))

    def rhs_config(self, v, eps=0.02):
        Nz, NJ = self.Nz, self.Ny + 5
        per = lambda f, d: torch.cat([f[:1], torch.roll(f[1:Nz], -d, 0), f[:1]])  # the Nz - 1 distinct planes

        def row(f, d):
            o = torch.zeros_like(f)
            o[:, 3:NJ - 3] = f[:, 3 + d:NJ - 3 + d]
            return o

        def d4(f, at, h):
            return (at(f, -2) - 8.0 * at(f, -1) + 8.0 * at(f, 1) - at(f, 2)) / (12.0 * h)

        def ko(f, at, h):
            q = -20.0 * f
            for d, w in ((1, 15.0), (2, -6.0), (3, 1.0)):
                q = q + w * (at(f, d) + at(f, -d))
            return q * (eps / (64.0 * h))

        al, be, sg, a = self.al, self.be, self.sg, self.al * self.sg
        dbe = self.d4_r(be)
        E = al * v[4] + be * v[1]
        H = (a * self.gtt) * v[2]
        H[:, :3] = -H[:, :3]
        H[:, NJ - 3:] = -H[:, NJ - 3:]
        r = [E, self.d4_r(al * v[4]) + be * self.d4_r(v[1]) + dbe * v[1], d4(E, row, self.dy), d4(E, per, self.dz),
             (self.d4_r((a * self.grr) * v[1]) + d4(H, row, self.dy) + d4((a * self.gpp) * v[3], per, self.dz)
              + be * self.d4_r(v[4] * sg)) / sg + dbe * v[4] - (al * self.m2) * v[0]]
        out = []
        for w in range(5):
            f, q = v[w], r[w].clone()
            rad = torch.zeros_like(f)
            rad[..., 3:-3] = sum(c * f[..., 3 + d:f.shape[-1] - 3 + d] for d, c in
                                 ((-3, 1.0), (-2, -6.0), (-1, 15.0), (0, -20.0), (1, 15.0), (2, -6.0), (3, 1.0)))
            q += rad * (eps / (64.0 * self.dx)) + ko(f, row, self.dy) + ko(f, per, self.dz)
            q[..., -1] = -(self.d4_r(f)[..., -1] + f[..., -1] / self.x[-1])
            q[0] = q[Nz] = 0.0
            q[:, :3] = 0.0
            q[:, NJ - 3:] = 0.0
            out.append(q)
        return out

    def fill_config(self, u, hold=None):
        for w in range(5):
            u[w][0] = u[w][self.Nz - 1]
            u[w][self.Nz] = u[w][1]
            self._poles(u[w], -1.0 if w == 2 else 1.0)
        return u


def _trapezium(n):
    w = torch.ones(n, dtype=torch.float64, device=DEV)
    w[0] = w[-1] = 0.5
    return w


def _legendre(L, th):
    """[l, m] -> norm P_lm(cos theta); on a pole row the m = 0 value is the norm squared, others 0"""
    x, s = torch.cos(th), torch.sin(th)
    P = torch.zeros((L + 1, L + 1, len(th)), dtype=torch.float64, device=DEV)
    pole = torch.abs(x) > 0.9999
    for m in range(L + 1):  # fully normalised recurrences
        P[m, m] = 1.0 / math.sqrt(4.0 * math.pi) if m == 0 else -math.sqrt((2 * m + 1) / (2.0 * m)) * s * P[m - 1, m - 1]
        for l in range(m + 1, L + 1):
            a = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
            b = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0))
            P[l, m] = a * (x * P[l - 1, m] - (b * P[l - 2, m] if l > m + 1 else 0.0))
    for l in range(L + 1):
        P[l, :, pole] = 0.0
        P[l, 0, pole] = (2 * l + 1) / (4.0 * math.pi)
    return P


def _sph_jl(l_max, x):
    """j_0 .. j_l_max at x (an array), by upward recurrence above l and Miller's downward one below"""
    out = np.zeros((l_max + 1,) + x.shape)
    j0 = np.sin(x) / x
    j1 = np.sin(x) / x ** 2 - np.cos(x) / x
    up = [j0, j1]
    for k in range(1, l_max):
        up.append((2 * k + 1) / x * up[k] - up[k - 1])
    top = l_max + 40 + int(math.sqrt(40.0 * (l_max + 1)))
    hi, cur, down = np.zeros_like(x), np.full_like(x, 1e-300), {}
    small = x <= l_max + 1.0
    xs = np.where(small, x, l_max + 1.0)
    for k in range(top, 0, -1):
        hi, cur = cur, (2 * k + 1) / xs * cur - hi
        big = np.abs(cur) > 1e200
        f = np.where(big, 1e-200, 1.0)
        hi, cur = hi * f, cur * f
        down = {q: v * f for q, v in down.items()}
        if k - 1 <= l_max:
            down[k - 1] = cur.copy()
    use0 = np.abs(j0) >= np.abs(j1)
    scale = np.where(use0, j0 / down[0], j1 / (down[1] if l_max >= 1 else hi))
    for l in range(l_max + 1):
        out[l] = np.where((x > l) & (l <= 1), up[l] if l < len(up) else j0,
                          np.where(x > l, up[l] if l < len(up) else j0, down[l] * scale))
    return out


def _jl(l, x):
    return _sph_jl(max(l, 1), np.asarray(x, np.float64))[l]


def _bessel(e, L, Nk):
    """normalised radial basis [l, n, shell] on the vertex radii, k = zeros of j_l over the outermost radius"""
    r = e.xmin + np.arange(e.Nx) * e.dx
    rmax = float(e.x[-1])
    zeros = np.pi * np.arange(1, Nk + L + 1)
    basis = np.zeros((L + 1, Nk, e.Nx))
    for l in range(L + 1):
        if l:
            lo, hi = zeros[:-1].copy(), zeros[1:].copy()
            flo = _jl(l, lo)
            for _ in range(80):
                mid = 0.5 * (lo + hi)
                fm = _jl(l, mid)
                same = (fm > 0) == (flo > 0)
                lo, flo, hi = np.where(same, mid, lo), np.where(same, fm, flo), np.where(same, hi, mid)
            zeros = 0.5 * (lo + hi)
        b = _jl(l, zeros[:Nk, None] / rmax * r[None, :])
        f = b ** 2 * r ** 2
        norm = np.sqrt(e.dx * (f.sum(1) - 0.5 * (f[:, 0] + f[:, -1])))
        basis[l] = b / norm[:, None]
    return r, basis


def _exact_of(c, u0=None, seed=0, **kw):
    x0, x1 = _domain(c["Nx"])
    e = _Exact(c["Nx"], c["Ny"], c["Nz"], x0, x1, m=c.get("m", 0.3), metric=c.get("metric", "Kerr_Schild"),
               bc=c.get("bc", "outflow"))
    u0 = _initial(c["Nx"], c["Ny"], c["Nz"], x0, x1, seed)
    return e, [u0[..., w].contiguous() for w in range(5)]


def _out(u):
    return torch.stack(u, dim=-1)


def _refine_exact(c, seed):
    x0, x1 = _domain(c["Nx"])
    lv, us = [], []
    dt = None
    for l in range(c["levels"]):
        if l == 0:
            nx, xm = c["Nx"], x1
        else:
            dx = lv[0].dx / 2 ** l
            nx = int((_radii(c)[l - 1] - x0) / dx)
            xm = x0 + nx * dx
        e = _Exact(nx, c["Ny"], c["Nz"], x0, xm, m=0.3, dt=dt and dt / 2 ** l)
        dt = dt or e.dt
        u0 = _initial(nx, c["Ny"], c["Nz"], x0, xm, seed)
        lv.append(e)
        us.append([u0[..., w].contiguous() for w in range(5)])
    nbuf, keep = 4, 8

    def planes(f, n):
        """the last nbuf planes of a fine level of n stored planes, from the coarse field f"""
        o = []
        for i in range(n - nbuf, n):
            a = i // 2
            o.append(f[..., a] if i % 2 == 0 else
                     (-f[..., a - 1] + 9.0 * f[..., a] + 9.0 * f[..., a + 1] - f[..., a + 2]) / 16.0)
        return torch.stack(o, dim=-1)

    def step(l, a0, da, old):
        mine = [f.clone() for f in us[l]]
        if l:
            n = lv[l].Nx + 5
            po, pn = [planes(f, n) for f in old], [planes(f, n) for f in us[l - 1]]

            def follow(v, at):
                for w in range(5):
                    v[w][..., -nbuf:] = (1.0 - (a0 + at * da)) * po[w] + (a0 + at * da) * pn[w]
            follow(us[l], 0.0)
        new = getattr(lv[l], c["stepper"])(us[l], **({"between": follow} if l else {}))
        if l:
            follow(new, 1.0)
        us[l] = new
        if l + 1 < c["levels"]:
            for sub in range(2):
                step(l + 1, 0.5 * sub, 0.5, mine)
            last = lv[l + 1].Nx + 4 - keep
            nc = last // 2 + 1
            for w in range(5):
                us[l][w][..., :nc] = us[l + 1][w][..., :2 * nc:2]

    for _ in range(c["steps"]):
        step(0, 0.0, 1.0, None)
    return [_out(u) for u in us]


def exact(case, seed):
    c = case
    if c["kind"] == "refine":
        return _refine_exact(c, seed)
    if c["kind"] == "batch":
        outs, alms = [], []
        for g in _members(c, seed):
            e, u = _exact_of(g, seed=g["seed"])
            for _ in range(c["steps"]):
                u = e.rk4(u)
            outs.append(_out(u))
            alms.append(e.alm_detectors(u))
        return [outs, alms]
    e, u = _exact_of(c, seed=seed)
    if c["kind"] == "spectral":
        shells = torch.stack([e.shell(u[0], i) for i in range(e.Nx)])
        a = e.alm(shells, c["L"])
        if not c["Nk"]:
            return a.cpu().numpy()
        r, basis = _bessel(e, c["L"], c["Nk"])
        w = np.full(e.Nx, e.dx)
        w[0] = w[-1] = 0.5 * e.dx
        return np.einsum("iml,lni->mln", a.cpu().numpy(), basis * (r * r * w))
    if c["kind"] == "config":
        e.fill_config(u)
        for _ in range(c["steps"]):
            u = e.rk4(u, rhs=e.rhs_config, fill=e.fill_config)
        return _out(u)
    if c["kind"] == "evolve":
        mass = []
        for _ in range(c["steps"]):
            u = e.pirk2(u)
            mass.append(e.mass(u))
        return [_out(u), np.array(mass)]
    for _ in range(c["steps"]):
        u = getattr(e, c["stepper"])(u)
    return [_out(u), e.mass(u), e.momentum(u), e.alm_detectors(u)]
