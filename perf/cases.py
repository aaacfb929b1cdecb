"""The work that users of the solver have it do, as cases to be timed and compared.

Every case goes through the Python front end (cflbm), as a user's program does:
channels stepped between two outputs, a channel whose force is read every step,
the reference-rule profiles, a batch of channels, a gradient, a dump and
restore.  `exact` forms the same outputs in 64 bits with plain torch.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cylinder-flow_gb300"))

import cflbm  # noqa: E402
from cflbm import adjoint as cflbm_adjoint  # noqa: E402

AMP = 1e-3  # amplitude of the seeded u_y perturbation every channel starts with
BYTES = {"fp64": 8, "fp32": 4, "fp16dev": 2}


def listed():
    return [
        # the small benchmark channel, its force read after every step (the
        # reference writes Cd and Cl to test.dat each step): the smallest calls
        channel("monitor2d_400x100_fp64", "monitor", 9, 400, 100, 1, "fp64", "fp64", 20, 20.0, 100.0),
        # the same channel run between two outputs: FP64 on a grid that stays in L2
        channel("channel2d_400x100_fp64", "channel", 9, 400, 100, 1, "fp64", "fp64", 400, 20.0, 100.0),
        # an odd-sized 2-D channel between no-slip walls, FP32 storage and collision
        channel("channel2d_1021x241_fp32", "channel", 9, 1021, 241, 1, "fp32", "fp32", 200, 24.0, 80.0,
                wall_y="noslip"),
        # the wide 2-D grid: FP32 streaming from HBM
        channel("wide2d_8192x1024_fp32", "channel", 9, 8192, 1024, 1, "fp32", "fp32", 20, 128.0, 150.0),
        # the headline: spanwise cylinder in the reference's own precision
        channel("cylinder3d_512x128x128_fp64", "channel", 27, 512, 128, 128, "fp64", "fp64", 10, 32.0,
                200.0, u0=0.04),
        # double-float arithmetic, ragged box with no-slip walls and a sphere
        channel("sphere3d_389x97x101_df64", "channel", 27, 389, 97, 101, "fp64", "df64", 10, 24.0, 150.0,
                u0=0.04, wall_y="noslip", wall_z="noslip", geom="sphere"),
        # the headline's channel in FP32
        channel("cylinder3d_512x128x128_fp32", "channel", 27, 512, 128, 128, "fp32", "fp32", 20, 32.0,
                200.0, u0=0.04),
        # the precision problem's sphere, FP16 deviations with stochastic rounding: the largest
        channel("sphere3d_768x384x384_fp16", "channel", 27, 768, 384, 384, "fp16dev", "fp32", 10, 64.0,
                300.0, u0=0.03, wall_z="freeslip", geom="sphere"),
        # the reference's own 3-D rules: what its main.cpp and input.in select
        dict(name="ref3d_257x97x97_fp64", kind="ref3d", nx=257, ny=97, nz=97, steps=20, u0=0.04,
             tau0=0.0192, storage="fp64", compute="fp64"),
        # many uneven channels at once, one launch sequence for all
        dict(name="batch_64_fp32", kind="batch", n=64, nx_max=1024, ny_max=256, steps=200, storage="fp32"),
        # drag gradient with respect to a porosity field, inlet speed and tau
        dict(name="adjoint_1024x256_fp32", kind="adjoint", nx=1024, ny=256, diam=32.0, re=100.0, u0=0.05,
             steps=600, every=100, begin=301, storage="fp32", wall_y="freeslip"),
        # a run dumped to the host, restored from there and continued, with its mass check
        channel("restart3d_256x64x64_fp32", "restart", 27, 256, 64, 64, "fp32", "fp32", 20, 16.0, 200.0,
                u0=0.04),
    ]


def channel(name, kind, lattice, nx, ny, nz, storage, compute, steps, diam, re, u0=0.05,
            wall_y="freeslip", wall_z="periodic", geom="cylinder"):
    c = dict(kind=kind, lattice=lattice, nx=nx, ny=ny, nz=nz, storage=storage, compute=compute,
             steps=steps, diam=diam, re=re, u0=u0, wall_y=wall_y, wall_z=wall_z, geom=geom)
    return dict(name=name, **c) if name else c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel2d", "channel2d", "channel3d", "channel3d", "channel3d", "monitor",
                       "ref2d", "ref3d", "batch", "adjoint", "restart"])
    form = rng.choice([("fp64", "fp64"), ("fp64", "fp64"), ("fp64", "df64"), ("fp64", "fp32"),
                       ("fp32", "fp32"), ("fp16dev", "fp32")])
    wall_y = rng.choice(["freeslip", "noslip", "periodic"])
    wall_z = rng.choice(["freeslip", "noslip", "periodic"])
    re, u0 = round(rng.uniform(40.0, 200.0), 1), round(rng.uniform(0.03, 0.05), 3)
    if kind in ("channel2d", "monitor"):
        ny = _log(rng, 64, 1024) if kind == "channel2d" else _log(rng, 64, 256)
        nx = min(8192, int(ny * rng.uniform(2.0, 8.0)))
        steps = max(10, min(400, int(2e8 / (nx * ny)))) if kind == "channel2d" else 20
        return channel(None, "monitor" if kind == "monitor" else "channel", 9, nx, ny, 1, *form, steps,
                       round(ny * rng.uniform(0.1, 0.2), 1), re, u0, wall_y)
    if kind in ("channel3d", "restart"):
        ny = _log(rng, 24, 200) if kind == "channel3d" else _log(rng, 24, 64)
        nz = max(8, int(ny * rng.uniform(0.5, 1.1)))
        nx = int(ny * rng.uniform(2.0, 4.0))
        steps = max(10, min(100, int(8e7 / (nx * ny * nz))))
        return channel(None, "restart" if kind == "restart" else "channel", 27, nx, ny, nz, *form, steps,
                       round(min(ny, nz) * rng.uniform(0.15, 0.3), 1), re, u0, wall_y, wall_z,
                       rng.choice(["cylinder", "sphere"]))
    if kind == "ref2d":
        nx, ny = _log(rng, 96, 1024), _log(rng, 40, 512)
        return dict(kind="ref2d", nx=nx, ny=ny, nz=1, steps=50, u0=u0, tau0=0.03, storage="fp64",
                    compute=rng.choice(["fp64", "df64", "fp32"]))
    if kind == "ref3d":
        n = _log(rng, 20, 90)
        return dict(kind="ref3d", nx=2 * n + rng.randrange(n), ny=n + rng.randrange(9), nz=n, steps=20,
                    u0=u0, tau0=0.0192, storage="fp64", compute=rng.choice(["fp64", "df64", "fp32"]))
    if kind == "batch":
        return dict(kind="batch", n=rng.randrange(4, 48), nx_max=rng.randrange(300, 1024),
                    ny_max=rng.randrange(80, 256), steps=rng.randrange(20, 200),
                    storage=rng.choice(["fp32", "fp16dev"]))
    ny = _log(rng, 48, 256)
    steps = rng.randrange(60, 300)
    return dict(kind="adjoint", nx=int(ny * rng.uniform(2.0, 4.0)), ny=ny, diam=round(0.14 * ny, 1), re=re,
                u0=u0, steps=steps, every=rng.choice([10, 25, 50, 100]), begin=1 + steps // 2,
                storage=rng.choice(["fp32", "fp64"]), wall_y=wall_y)


# ---- inputs --------------------------------------------------------------------------
def _channel_kw(case, seed):
    """Solver keywords of a channel: the body a quarter of the way down the box."""
    return dict(lattice=case["lattice"], nx=case["nx"], ny=case["ny"], nz=case["nz"],
                storage=case["storage"], compute=case["compute"], u0=case["u0"],
                tau0=3.0 * case["u0"] * case["diam"] / case["re"], wall_y=case["wall_y"],
                wall_z=case["wall_z"], geom=case["geom"], cx=case["nx"] / 4.0, cy=case["ny"] / 2.0,
                cz=case["nz"] / 2.0, diam=case["diam"], perturb_amp=AMP, seed=int(seed))


def _batch_kws(case, seed):
    rng = np.random.default_rng(2025)  # the channels; the seed draws their perturbations
    kws = []
    for k in range(case["n"]):
        nx = int(rng.integers(256, case["nx_max"] + 1))
        ny = int(rng.integers(64, case["ny_max"] + 1))
        if k % 2 == 0:  # every other channel in whole 32-cell tiles
            nx, ny = nx // 32 * 32, ny // 32 * 32
        d = float(rng.uniform(8.0, 24.0))
        re = float(rng.uniform(40.0, 200.0))
        kws.append(dict(lattice=9, nx=nx, ny=ny, tau0=3.0 * 0.05 * d / re, u0=0.05, wall_y="freeslip",
                        geom="cylinder", cx=4.0 * d, cy=ny / 2.0, diam=d, perturb_amp=AMP,
                        storage=case["storage"], compute="fp32", seed=1000 * int(seed) + k))
    return kws


def _adjoint_inputs(case, seed):
    """(solver keywords, porosity field, tau): a smooth seeded porosity on a box
    around the cylinder, in FP32 as an optimiser holds it."""
    nx, ny, d = case["nx"], case["ny"], case["diam"]
    cx, cy = nx / 5.0, ny / 2.0
    kw = dict(lattice=9, nx=nx, ny=ny, geom="cylinder", cx=cx, cy=cy, diam=d, wall_y=case["wall_y"],
              perturb_amp=AMP, seed=int(seed), storage=case["storage"], compute=case["storage"])
    rng = np.random.default_rng(int(seed))
    X, Y = np.meshgrid(np.arange(nx), np.arange(ny))
    a = np.zeros((ny, nx))
    for _ in range(8):
        x0, y0, w = rng.uniform(cx - 2 * d, cx + 2 * d), rng.uniform(cy - 2 * d, cy + 2 * d), \
            rng.uniform(d / 4, 3 * d / 4)
        a += rng.uniform(0.5, 1.0) * np.exp(-((X - x0) ** 2 + (Y - y0) ** 2) / (2.0 * w * w))
    a *= (abs(X - cx) < 2 * d) & (abs(Y - cy) < 2 * d)
    return kw, (a / a.max()).astype(np.float32), 0.5 + 3.0 * case["u0"] * d / case["re"]


def _ref_ran(case, seed):
    g = 2 if case["kind"] == "ref2d" else 3
    shape = (case["nx"] + 2 * g, case["ny"] + 2 * g) + ((case["nz"] + 2 * g,) if g == 3 else ())
    return np.random.default_rng(int(seed)).integers(0, 100, size=shape).astype(np.int32)


def _fields(shape, n):
    return [torch.empty(shape, dtype=torch.float64, device="cuda") for _ in range(n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("channel", "monitor", "restart"):
        s = cflbm.Solver(force_history=1024, **_channel_kw(case, seed))
        return dict(kind=kind, steps=case["steps"], solver=s,
                    fields=_fields(s.shape, 3 if case["lattice"] == 9 else 4))
    if kind in ("ref2d", "ref3d"):
        s = cflbm.Solver(lattice=9 if kind == "ref2d" else 27, nx=case["nx"], ny=case["ny"],
                         nz=case["nz"], profile=kind, tau0=case["tau0"], u0=case["u0"],
                         storage=case["storage"], compute=case["compute"], force_history=1024,
                         ref_ran=_ref_ran(case, seed))
        return dict(kind="channel", steps=case["steps"], solver=s,
                    fields=_fields(s.shape, 3 if kind == "ref2d" else 4))
    if kind == "batch":
        kws = _batch_kws(case, seed)
        cells = [k["nx"] * k["ny"] for k in kws]
        at = np.concatenate([[0], np.cumsum(cells)])
        flat = [torch.empty(int(at[-1]), dtype=torch.float64, device="cuda") for _ in range(3)]
        b = cflbm.Batch([dict(k, force_history=1024) for k in kws])
        return dict(kind=kind, steps=case["steps"], batch=b, inst=[b.instance(k) for k in range(case["n"])],
                    fields=flat, parts=[[t[int(at[k]):int(at[k + 1])] for t in flat]
                                        for k in range(case["n"])])
    kw, alpha, tau = _adjoint_inputs(case, seed)
    return dict(kind="adjoint", case=kw, alpha=torch.from_numpy(alpha).cuda(),
                u_in=torch.tensor(case["u0"], dtype=torch.float32),
                tau=torch.tensor(tau, dtype=torch.float32), steps=case["steps"], every=case["every"],
                window=(case["begin"], case["steps"]))


# ---- one pass ------------------------------------------------------------------------
def _macros(s, t):
    s.macros_device(t[0], t[1], t[2] if len(t) == 4 else None, t[-1])


def run(state):
    kind, n = state["kind"], state["steps"]
    if kind == "channel":  # steps, then the fields and the force of every step
        s = state["solver"]
        s.step(n)
        _macros(s, state["fields"])
        return {"fields": state["fields"], "force": s.force_history(n)}
    if kind == "monitor":  # the force read on the host after every step
        s = state["solver"]
        rows = []
        for _ in range(n):
            s.step(1)
            rows.append(np.concatenate(s.forces()))
        _macros(s, state["fields"])
        return {"fields": state["fields"], "force": np.stack(rows)}
    if kind == "restart":  # dump, restore, mass check, continue
        s = state["solver"]
        f = s.get_f()
        s.set_f(f, steps_done=0)
        mass, momentum = s.mass()
        s.step(n)
        _macros(s, state["fields"])
        return {"f": f, "mass": mass, "momentum": momentum, "fields": state["fields"],
                "force": s.force_history(n)}
    if kind == "batch":  # every channel's fields and forces after the steps
        state["batch"].step(n)
        for s, part in zip(state["inst"], state["parts"]):
            s.macros_device(part[0], part[1], None, part[2])
        return {"fields": state["fields"], "force": np.stack([s.force_history(n) for s in state["inst"]])}
    # adjoint: the objective and its gradients, as an optimiser asks for them
    alpha = state["alpha"].detach().requires_grad_(True)
    u_in = state["u_in"].detach().requires_grad_(True)
    tau = state["tau"].detach().requires_grad_(True)
    J = cflbm_adjoint.drag_objective(alpha, u_in, tau, state["case"], n, state["every"], state["window"])
    J.backward()
    return {"J": J.detach(), "alpha": alpha.grad, "u_in": u_in.grad, "tau": tau.grad}


def work(case):
    """Bytes and operations of a pass: every step reads and writes each population
    once; u, v, (w,) p and the dumped state are written once."""
    kind = case["kind"]
    if kind == "batch":
        q, es, cells, out = 9, BYTES[case["storage"]], sum(k["nx"] * k["ny"] for k in _batch_kws(case, 0)), 24
    elif kind == "adjoint":
        q, es, cells, out = 9, BYTES[case["storage"]], case["nx"] * case["ny"], 4
    else:
        q = 9 if case.get("lattice", 27 if kind == "ref3d" else 9) == 9 else 27
        es, cells, out = BYTES[case["storage"]], case["nx"] * case["ny"] * case["nz"], 24 if q == 9 else 32
    per_step = 2.0 * q * es
    ops = 80.0 if q == 9 else 220.0
    if kind == "adjoint":  # the reverse step reads a state and the co-state and writes the co-state
        per_step, ops = 5.0 * q * es, 250.0
    if kind == "restart":  # the dump, the restore and the mass check
        out += q * (8.0 + es) * 2.0 + q * es
    return {"bytes": cells * (per_step * case["steps"] + out), "flops": cells * ops * case["steps"]}


# ---- the same in 64 bits ---------------------------------------------------------------
E9 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
E27 = [(0, 0, 0)] + [s for p in [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1),
                                 (0, 1, 1), (0, 1, -1), (1, 1, 1), (1, -1, 1), (1, 1, -1), (1, -1, -1)]
                     for s in (p, tuple(-v for v in p))]


class _Exact:
    """The channel in FP64 torch: f[Q][nz, ny, nx], the post-collision state."""

    def __init__(self, kw, keep=True):
        self.E = E9 if kw["lattice"] == 9 else E27
        c0, r = (4.0 / 9.0, 4.0) if kw["lattice"] == 9 else (8.0 / 27.0, 4.0)
        self.w = [c0 / r ** sum(abs(v) for v in e) for e in self.E]
        self.opp = [self.E.index(tuple(-v for v in e)) for e in self.E]
        self.nz, self.ny, self.nx = (1 if kw["lattice"] == 9 else kw["nz"]), kw["ny"], kw["nx"]
        self.walls = {1: kw.get("wall_y", "freeslip"), 2: kw.get("wall_z", "periodic")}
        dev = "cuda"
        x = torch.arange(self.nx, dtype=torch.float64, device=dev).view(1, 1, -1)
        y = torch.arange(self.ny, dtype=torch.float64, device=dev).view(1, -1, 1)
        z = torch.arange(self.nz, dtype=torch.float64, device=dev).view(-1, 1, 1)
        d2 = (x - kw["cx"]) ** 2 + (y - kw["cy"]) ** 2 + (0.0 * z)
        if kw["geom"] == "sphere":
            d2 = d2 + (z - kw["cz"]) ** 2
        self.solid = d2 <= 0.25 * kw["diam"] ** 2
        self.keep = [None] * len(self.E) if keep else None
        cells = np.arange(self.nz * self.ny * self.nx, dtype=np.uint64)
        with np.errstate(over="ignore"):
            h = np.uint64(kw["seed"]) + cells * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0x9E3779B97F4A7C15)
            h = (h ^ (h >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            h = (h ^ (h >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            h = h ^ (h >> np.uint64(31))
        r01 = (h >> np.uint64(11)).astype(np.float64) / 2.0 ** 53
        v0 = torch.from_numpy(kw["perturb_amp"] * (2.0 * r01 - 1.0)).to(dev).view(self.nz, self.ny, self.nx)
        self.v0 = torch.where(self.solid, 0.0, v0)

    def feq(self, i, rho3, u):
        eu = sum(e * c for e, c in zip(self.E[i], u) if e) if any(self.E[i]) else 0.0 * u[0]
        uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        return self.w[i] * (rho3 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu)

    def start(self, u_in, omega, alpha=None):
        z = torch.zeros_like(self.v0)
        u = [torch.where(self.solid, z, z + u_in), self.v0, z]
        f = [self.feq(i, z, u) for i in range(len(self.E))]
        return f if alpha is None else self.collide(f, z, u, omega, alpha)

    def collide(self, g, rho3, u, omega, alpha=None):
        if alpha is not None:
            u = [(1.0 - alpha) * c for c in u]
        return [gi - omega * (gi - self.feq(i, rho3, u)) for i, gi in enumerate(g)]

    def source(self, i):
        """(index into the flat populations [Q, cells], inlet mask, solid links)."""
        if self.keep is not None and self.keep[i] is not None:
            return self.keep[i]
        e, dev, n = self.E[i], "cuda", (self.nx, self.ny, self.nz)
        at = [torch.arange(n[d], device=dev) - e[d] for d in range(3)]
        out = [(a < 0) | (a >= n[d]) for d, a in enumerate(at)]
        pop = {}
        bounce = [torch.zeros(n[d], dtype=torch.bool, device=dev) for d in range(3)]
        flip = [torch.zeros(n[d], dtype=torch.bool, device=dev) for d in range(3)]
        for d in (1, 2):
            if self.walls[d] == "periodic":
                at[d] = at[d] % n[d]
            elif self.walls[d] == "freeslip":
                flip[d] = out[d]
                at[d] = torch.where(out[d], at[d] + e[d], at[d])
            else:
                bounce[d] = out[d]
                at[d] = at[d].clamp(0, n[d] - 1)
        for fy in (0, 1):
            for fz in (0, 1):
                pop[fy, fz] = self.E.index((e[0], -e[1] if fy else e[1], -e[2] if fz else e[2]))
        X, Y, Z = (lambda v: v.view(1, 1, -1)), (lambda v: v.view(1, -1, 1)), (lambda v: v.view(-1, 1, 1))
        j = torch.where(Y(flip[1]), torch.where(Z(flip[2]), pop[1, 1], pop[1, 0]),
                        torch.where(Z(flip[2]), pop[0, 1], pop[0, 0]))
        inlet = X(at[0] < 0)
        sx = at[0].clamp(0, self.nx - 1)
        wall = Y(bounce[1]) | Z(bounce[2])
        src = (Z(at[2]) * self.ny + Y(at[1])) * self.nx + X(sx)
        link = self.solid.view(-1)[src] & ~inlet & ~wall
        N = self.nx * self.ny * self.nz
        here = torch.arange(N, device=dev).view(self.nz, self.ny, self.nx) + self.opp[i] * N
        idx = torch.where(link | wall, here, src + j * N)
        got = (idx, inlet & ~wall & ~link, link)
        if self.keep is not None:
            self.keep[i] = got
        return got

    def pull(self, f, u_in):
        flat = torch.stack(f).view(-1)
        zero = torch.zeros((), dtype=torch.float64, device="cuda")
        u = [zero + u_in, zero, zero]
        return [f[0]] + [torch.where(self.source(i)[1], self.feq(i, zero, u), flat[self.source(i)[0]])
                         for i in range(1, len(self.E))]

    def force(self, f):
        F = [torch.zeros((), dtype=torch.float64, device="cuda") for _ in range(3)]
        for i in range(1, len(self.E)):
            m = (2.0 * f[self.opp[i]] * (self.source(i)[2] & ~self.solid)).sum()
            F = [a - e * m for a, e in zip(F, self.E[i])]
        return torch.stack(F)

    def moments(self, g):
        rho3 = sum(g)
        u = [sum(e[d] * gi for e, gi in zip(self.E, g) if e[d]) if self.nz > 1 or d < 2 else 0.0 * rho3
             for d in range(3)]
        return torch.where(self.solid, 0.0, rho3), [torch.where(self.solid, 0.0, c) for c in u]

    def steps(self, f, n, u_in, omega):
        """(state, force rows, rho3, u) after n steps."""
        rows, rho3, u = [], None, None
        for _ in range(n):
            rows.append(self.force(f))
            g = self.pull(f, u_in)
            rho3, u = self.moments(g)
            f = self.collide(g, rho3, u, omega)
        return f, torch.stack(rows), rho3, u


def _exact_channel(case, seed):
    kw = _channel_kw(case, seed)
    ex = _Exact(kw, keep=case["nx"] * case["ny"] * case["nz"] < 3e7)
    omega = 1.0 / (kw["tau0"] + 0.5)
    f0 = ex.start(kw["u0"], omega)
    f, rows, rho3, u = ex.steps(f0, case["steps"], kw["u0"], omega)
    fields = [u[0], u[1]] + ([u[2]] if kw["lattice"] == 27 else []) + [rho3 / 3.0]
    rows = rows.cpu().numpy()
    if case["kind"] == "monitor":
        rows = np.concatenate([rows, 2.0 * rows[:, :2] / (kw["u0"] ** 2 * case["diam"])], axis=1)
    out = {"fields": fields, "force": rows}
    if case["kind"] == "restart":
        fluid = ~ex.solid
        out["f"] = torch.stack(f0)
        out["mass"] = float(((1.0 + sum(f0)) * fluid).sum())
        out["momentum"] = np.array([float((sum(e[d] * fi for e, fi in zip(ex.E, f0)) * fluid).sum())
                                    for d in range(3)])
    return out


def _exact_ref(case, seed):
    """The reference's rules: face passes and the solid fill on one ghosted
    array, plain pull, Poiseuille inlet and p = 0 outlet overrides."""
    d3 = case["kind"] == "ref3d"
    nx, ny, nz, u0 = case["nx"], case["ny"], case["nz"], case["u0"]
    E = E27 if d3 else E9
    w = [(8.0 / 27.0 if d3 else 4.0 / 9.0) / 4.0 ** sum(abs(v) for v in e) for e in E]
    opp = [E.index(tuple(-v for v in e)) for e in E]
    Q, G, Gz = len(E), (3 if d3 else 2), (3 if d3 else 0)
    omega = 1.0 / (case["tau0"] + 0.5)
    t64 = dict(dtype=torch.float64, device="cuda")
    X = (torch.arange(nx + 2 * G, **t64) - G).view(1, 1, -1)
    Y = (torch.arange(ny + 2 * G, **t64) - G).view(1, -1, 1)
    Z = (torch.arange(nz + 2 * Gz, **t64) - Gz).view(-1, 1, 1)
    ran = torch.from_numpy(_ref_ran(case, seed)).to("cuda").double()
    if d3:
        c = (nx - 1) // 8
        solid = (X - c) ** 2 + (Y - c) ** 2 + (Z - c) ** 2 <= ((nx - 1) / 64.0) ** 2
        u = (u0 * 4.0 * Z * (nz - 1 - Z) / (nz - 1) ** 2) * ~solid * (1.0 + ran.permute(2, 1, 0) * 0.001)
        inlet = (u0 * 4.0 * Z * (nz - 1 - Z) / (nz - 1) ** 2)[G:G + nz, :, 0].expand(nz, ny)
    else:
        solid = (X - 0.5 * (nx - 1)) ** 2 + (Y - 0.5 * (ny - 1)) ** 2 + 0 * Z <= (0.03125 * (nx - 1) / 2.0) ** 2
        u = (u0 * 4.0 * Y * (ny - 1 - Y) / (ny - 1) ** 2) * ~solid * (0.9 + ran.t()[None] * 0.002)
        inlet = (u0 * 4.0 * Y * (ny - 1 - Y) / (ny - 1) ** 2)[:, G:G + ny, 0]

    def feq(i, rho3, u, v, z):
        eu = E[i][0] * u + E[i][1] * v + E[i][2] * z
        return w[i] * (rho3 + 3.0 * eu + 4.5 * eu * eu - 1.5 * (u * u + v * v + z * z))

    zero = torch.zeros_like(u)
    f = torch.stack([feq(i, zero, u, zero, zero) for i in range(Q)])
    sl = (slice(Gz, Gz + nz), slice(G, G + ny), slice(G, G + nx))
    solid = solid[sl]
    n, ghost = (nx, ny, nz), (G, G, Gz)

    def layer(axis, v, shift=(0, 0, 0)):
        """Index of layer v of an axis over the interior plus one ring, shifted."""
        ix = [None, None, None]
        for d in range(3):
            if d == axis:
                ix[d] = v + ghost[d]
            elif d == 2 and not d3:
                ix[d] = slice(0, 1)
            else:
                ix[d] = slice(ghost[d] - 1 + shift[d], ghost[d] + n[d] + 1 + shift[d])
        return ix[2], ix[1], ix[0]

    def wall(axis, low):
        for i in range(Q):
            if (E[i][axis] > 0) if low else (E[i][axis] < 0):
                f[i][layer(axis, -1 if low else n[axis])] = \
                    f[opp[i]][layer(axis, 1 if low else n[axis] - 2, [2 * v for v in E[i]])].clone()

    def ends():
        for i in range(Q):
            if E[i][0] > 0:
                f[i][layer(0, -1)] = f[i][layer(0, 0)].clone()
            if E[i][0] < 0:
                f[i][layer(0, nx)] = f[i][layer(0, nx - 1, E[i])].clone()

    links = []
    pad = torch.nn.functional.pad(solid.double(), (1, 1, 1, 1, 1, 1), value=2.0)
    for k in range(1, Q):
        e = E[k]
        near = pad[1 + e[2]:1 + e[2] + nz, 1 + e[1]:1 + e[1] + ny, 1 + e[0]:1 + e[0] + nx]
        s = torch.nonzero(solid & (near == 0.0))
        links.append([s[:, d] + g for d, g in zip(range(3), (Gz, G, G))])
    rows = []
    for _ in range(case["steps"]):
        if d3:
            for axis in (1, 2):
                wall(axis, True)
                wall(axis, False)
            ends()
        else:
            ends()
            wall(1, True)
            wall(1, False)
        F = [0.0, 0.0, 0.0]
        new = []
        for k in range(1, Q):
            (z, y, x), e = links[k - 1], E[k]
            v = f[opp[k]][z + 2 * e[2], y + 2 * e[1], x + 2 * e[0]]
            m = (f[opp[k]][z + e[2], y + e[1], x + e[0]] + v).sum()
            F = [a - c * m for a, c in zip(F, e)]
            new.append(v)
        for k in range(1, Q):
            z, y, x = links[k - 1]
            f[k][z, y, x] = new[k - 1]
        rows.append(torch.stack([a + torch.zeros((), **t64) for a in F]))
        g = [f[i][Gz - e[2]:Gz - e[2] + nz, G - e[1]:G - e[1] + ny, G - e[0]:G - e[0] + nx].clone()
             for i, e in enumerate(E)]
        rho3 = torch.where(solid, 0.0, sum(g))
        m = [torch.where(solid, 0.0, sum(e[d] * gi for e, gi in zip(E, g))) for d in range(3)]
        m[0][..., 0], m[1][..., 0], m[2][..., 0], rho3[..., nx - 1] = inlet, 0.0, 0.0, 0.0
        for i in range(Q):
            f[i][sl] = g[i] - omega * (g[i] - feq(i, rho3, *m))
    return {"fields": m[:3 if d3 else 2] + [rho3 / 3.0], "force": torch.stack(rows).cpu().numpy()}


def _exact_adjoint(case, seed):
    kw, alpha, tau = _adjoint_inputs(case, seed)
    ex = _Exact(kw)
    t64 = dict(dtype=torch.float64, device="cuda")
    par = [torch.from_numpy(alpha).to(**t64)[None], torch.tensor(np.float32(case["u0"]), **t64),
           torch.tensor(np.float32(tau), **t64)]
    n, first = case["steps"], case["begin"]
    weight = 1.0 / (n - first + 1)

    def leaves():
        return [p.clone().requires_grad_(True) for p in par]

    def step(f, a, u_in, tau):
        g = ex.pull(f, u_in)
        rho3, u = ex.moments(g)
        return ex.collide(g, rho3, u, 1.0 / tau, a)

    states, J = [], 0.0
    with torch.no_grad():
        f = ex.start(par[1], 1.0 / par[2], par[0])
        for t in range(1, n + 1):
            states.append(f)
            if t >= first:
                J += weight * float(ex.force(f)[0])
            f = step(f, *par)
    grad, lam = [torch.zeros_like(p) for p in par], None
    for t in range(n, 0, -1):  # lam = dJ/ds_t, from the force of step t and the step to s_{t+1}
        s = [c.clone().requires_grad_(True) for c in states.pop()]
        p = leaves()
        total = (ex.force(s)[0] * weight) if t >= first else 0.0
        if lam is not None:
            total = total + sum((a * b).sum() for a, b in zip(lam, step(s, *p)))
        if isinstance(total, float):
            continue
        got = torch.autograd.grad(total, s + p, allow_unused=True)
        lam = [torch.zeros_like(c) if g is None else g for c, g in zip(s, got)]
        grad = [a if g is None else a + g for a, g in zip(grad, got[len(s):])]
    p = leaves()
    total = sum((a * b).sum() for a, b in zip(lam, ex.start(p[1], 1.0 / p[2], p[0])))
    got = torch.autograd.grad(total, p, allow_unused=True)
    grad = [a if g is None else a + g for a, g in zip(grad, got)]
    return {"J": torch.tensor(J, dtype=torch.float64), "alpha": grad[0][0], "u_in": grad[1], "tau": grad[2]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("channel", "monitor", "restart"):
        return _exact_channel(case, seed)
    if kind in ("ref2d", "ref3d"):
        return _exact_ref(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    fields, force = [[], [], []], []
    for kw in _batch_kws(case, seed):
        ex = _Exact(dict(kw, cz=0.0))
        omega = 1.0 / (kw["tau0"] + 0.5)
        _, rows, rho3, u = ex.steps(ex.start(kw["u0"], omega), case["steps"], kw["u0"], omega)
        for t, v in zip(fields, (u[0], u[1], rho3 / 3.0)):
            t.append(v.reshape(-1))
        force.append(rows.cpu().numpy())
    return {"fields": [torch.cat(t) for t in fields], "force": np.stack(force)}
