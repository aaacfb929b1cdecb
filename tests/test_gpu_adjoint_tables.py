"""The reverse sweep's tables and sums against automatic differentiation.

A dense FP64 restatement of the channel step (one gather per population from the
rules of every cell) is differentiated by torch on small boxes with bodies on the
walls, the inlet, the outlet and alone; checkpoint spacings cover direct and
captured segments.  Tolerances: FP64 1e-9 of the largest gradient (12 steps of
round-off); FP32 2e-3 (forward and reverse in FP32, 2^-24 per operation over 12
steps, against gradients summed with cancellation).
"""
import numpy as np
import pytest
import torch

from test_gpu_fixed_point import E9

pytestmark = pytest.mark.gpu
W9 = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
OPP = [E9.index(tuple(-v for v in e)) for e in E9]


def gather(solid, wall):
    """Per population: flat source index into f[9, ny, nx], inlet mask, link mask."""
    ny, nx = solid.shape
    idx, inlet, link = (np.zeros((9, ny, nx), int) for _ in range(3))
    for i, e in enumerate(E9):
        for y in range(ny):
            for x in range(nx):
                sx, sy, j, bb = x - e[0], y - e[1], i, False
                if not 0 <= sy < ny:
                    if wall == "periodic":
                        sy %= ny
                    elif wall == "freeslip":
                        j, sy = E9.index((e[0], -e[1], 0)), y
                    else:
                        bb = True
                if i and not bb and sx >= 0 and solid[min(max(sy, 0), ny - 1), min(sx, nx - 1)]:
                    bb = True
                    link[i, y, x] = 1
                if i and bb:
                    sx, sy, j = x, y, OPP[i]
                elif sx < 0:
                    inlet[i, y, x], sx = 1, 0
                idx[i, y, x] = (j * ny + sy) * nx + min(sx, nx - 1)
    return (torch.from_numpy(a) for a in (idx, inlet.astype(bool), link.astype(bool)))


def reference(solid, wall, v0, alpha, u_in, tau, steps, window, axis):
    ny, nx = solid.shape
    idx, inlet, link = gather(solid, wall)
    fluid = torch.from_numpy(~solid)
    w = torch.from_numpy(W9).view(9, 1, 1)
    ex, ey = (torch.tensor([e[d] for e in E9], dtype=torch.float64).view(9, 1, 1) for d in (0, 1))

    def feq(rho3, ux, uy):
        eu = ex * ux + ey * uy
        return w * (rho3 + 3 * eu + 4.5 * eu * eu - 1.5 * (ux * ux + uy * uy))

    zero = torch.zeros(1, ny, nx, dtype=torch.float64)
    om, damp = 1.0 / tau, (1.0 - alpha)[None]
    ux, uy = torch.where(fluid, u_in, 0.0)[None], torch.from_numpy(np.where(solid, 0.0, v0))[None]
    f0 = feq(zero, ux, uy)
    f = f0 - om * (f0 - feq(zero, damp * ux, damp * uy))
    J = 0.0
    e = ex if axis == 0 else ey
    for t in range(1, steps + 1):
        if window[0] <= t <= window[1]:  # sum over links of 2 f_opp(i) e_opp(i)
            J = J - (2.0 * f[OPP] * e * (link & fluid)).sum() / (window[1] - window[0] + 1)
        g = torch.where(inlet, feq(zero, u_in, zero), f.reshape(-1)[idx])
        rho3 = torch.where(fluid, g.sum(0), 0.0)[None]
        ux = damp * torch.where(fluid, (ex * g).sum(0), 0.0)[None]
        uy = damp * torch.where(fluid, (ey * g).sum(0), 0.0)[None]
        f = g - om * (g - feq(rho3, ux, uy))
    return J


def bodies(name, ny, nx):
    s = np.zeros((ny, nx), np.uint8)
    if name == "disk":
        y, x = np.mgrid[0:ny, 0:nx]
        s[(x - nx * 0.4) ** 2 + (y - ny / 2) ** 2 <= 9] = 1
    elif name == "edges":   # on both walls, at the inlet, at the outlet, a thin plate
        s[0:2, 10:13] = s[ny - 1:, 20:22] = s[6:8, 0:1] = s[3:5, nx - 1:] = 1
        s[9, 15:19] = 1
    elif name == "porous":
        s[:] = np.random.default_rng(4).random((ny, nx)) < 0.12
    return s


@pytest.mark.parametrize("every", [5, 1])
@pytest.mark.parametrize("wall", ["freeslip", "noslip", "periodic"])
@pytest.mark.parametrize("body", ["disk", "edges", "porous"])
def test_gradients_match_autodiff(cuda, body, wall, every):
    from cflbm import Solver
    ny, nx, steps, window = 14, 37, 12, (4, 12)
    solid = bodies(body, ny, nx)
    rng = np.random.default_rng(1)
    alpha = (0.3 * rng.random((ny, nx))).astype(np.float32).astype(np.float64)
    u_in, tau = 0.04, 0.62
    for axis, objective in enumerate(("drag", "lift")):
        got = {}
        for form in ("fp64", "fp32"):
            with Solver(lattice=9, nx=nx, ny=ny, wall_y=wall, solid=solid, u0=u_in, tau0=tau - 0.5,
                        perturb_amp=1e-3, seed=9, alpha=alpha, storage=form, compute=form,
                        force_history=steps) as s:
                v0 = s.macros()[1].reshape(ny, nx)
                got[form] = s.adjoint(steps, every, window, objective)
        p = [torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in (u_in, tau)]
        a = torch.from_numpy(alpha).requires_grad_(True)
        J = reference(solid.astype(bool), wall, v0, a, p[0], p[1], steps, window, axis)
        J.backward()
        ref = {"J": float(J.detach()), "dJ_dalpha": a.grad.numpy() * (solid == 0),
               "dJ_du_in": float(p[0].grad), "dJ_dtau": float(p[1].grad)}
        for form, tol in (("fp64", 1e-9), ("fp32", 2e-3)):
            for k in ref:
                g = got[form][k] * (solid == 0) if k == "dJ_dalpha" else got[form][k]
                scale = max(np.abs(ref[k]).max(), 1e-3 * abs(ref["dJ_du_in"]))
                assert np.abs(g - ref[k]).max() <= tol * scale, (objective, form, k)
