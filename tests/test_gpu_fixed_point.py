"""The FP64 collision in block fixed point against one step in extended precision.

Error bound: the populations enter and leave in units of 2^-54 of the cell's
largest |f_i / w_i|; summing the worst case of every rounding (inputs, moments,
6 products, 2 constants, the product with 1 - omega) gives 16 such units, plus
the final rounding to FP64: 12 x 2^-53.  Cells outside the format (|f_i / w_i|
large, infinities, NaNs) take FP64 operations: 64 x 2^-53 covers their chain of
about 60 roundings.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E9 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]
E27 = [(0, 0, 0)] + [s for p in [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1),
                                 (0, 1, 1), (0, 1, -1), (1, 1, 1), (1, -1, 1), (1, 1, -1), (1, -1, -1)]
                     for s in (p, tuple(-v for v in p))]


def one_step(f, E, w, omega, damp=1):
    """(next state, pulled state) of a periodic box in extended precision."""
    g = np.stack([np.roll(f[i], e[::-1], (0, 1, 2)) for i, e in enumerate(E)]).astype(np.longdouble)
    rho3 = g.sum(axis=0)
    u = [sum(e[d] * gi for e, gi in zip(E, g) if e[d]) for d in range(3)]
    u = [c if isinstance(c, np.ndarray) else 0 * rho3 for c in u]
    u = [damp * c for c in u]
    usq = sum(c * c for c in u)
    out = []
    for i, e in enumerate(E):
        eu = sum(e[d] * u[d] for d in range(3))
        feq = w[i] * (rho3 + 3 * eu + np.longdouble(4.5) * eu * eu - np.longdouble(1.5) * usq)
        out.append(g[i] - np.longdouble(omega) * (g[i] - feq))
    return np.stack(out), g


def states(E, w, shape):
    """Random states of every size the format meets, one size per z or y layer:
    ordinary flows, tiny and zero ones, cells of mixed size, cells beyond it."""
    rng = np.random.default_rng(5)
    f = rng.normal(size=(len(E),) + shape) * w.reshape(-1, 1, 1, 1).astype(float)
    amp = np.array([0.05, 0.3, 1e-3, 1e-9, 1e-200, 0.0, 3.0, 40.0])
    rows = amp[np.arange(shape[1]) * len(amp) // shape[1]].reshape(1, -1, 1)
    f *= rows
    f[rng.integers(0, len(E)), :, 1, :] *= 1e-7          # one population far below the others
    f[:, :, :, ::7] *= rng.choice([1.0, 1e-3, 0.0], size=f[:, :, :, ::7].shape)
    return f


@pytest.mark.parametrize("layout", ["rows", "soa"])
@pytest.mark.parametrize("tau0", [1e-4, 0.0192, 0.6])
@pytest.mark.parametrize("lattice,dims", [(9, (67, 48, 1)), (27, (67, 32, 9)), (27, (64, 40, 4))])
def test_one_step_error(cuda, lattice, dims, tau0, layout):
    from cflbm import Solver
    E = E9 if lattice == 9 else E27
    w = np.array([(np.longdouble(4) / 9 if lattice == 9 else np.longdouble(8) / 27)
                  / np.longdouble(4) ** sum(map(abs, e)) for e in E])
    nx, ny, nz = dims
    f = states(E, w, (nz, ny, nx))
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=tau0, u0=0.04, wall_y="periodic",
                wall_z="periodic", geom="none", layout=layout) as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
        mac = [np.asarray(m).reshape(f.shape[1:]) for m in s.macros()]
    ref, g = one_step(f, E, w, 1.0 / (tau0 + 0.5))
    ins = (slice(None), slice(None), slice(1, nx - 1))   # the inlet and outlet columns have rules
    scale = np.abs(g / w.reshape(-1, 1, 1, 1)).max(axis=0)
    err = np.abs((got - ref) / w.reshape(-1, 1, 1, 1)).max(axis=0).astype(float)
    # largest |f / w| of a cell the format covers: |f_i 2^-k_i| < 1/4, w = W 2^k
    W = 1.0 / 27.0 if lattice == 27 else 1.0 / 9.0
    inside = scale < 0.2 / W
    # the u^2 terms of cells far beyond it scale with (f / w)^2
    tol = np.where(inside, 12.0, 64.0 * (1.0 + scale)) * 2.0 ** -53 * scale
    tol = np.maximum(tol, 2.0 ** -940).astype(float)
    assert (err[ins] <= tol[ins]).all(), float((err[ins] / tol[ins]).max())
    assert inside[ins].any() and (~inside[ins]).any()
    p = g.sum(axis=0) / 3
    assert (np.abs(mac[3] - p)[ins] <= 32 * 2.0 ** -53 * scale[ins] + 2.0 ** -940).all()


@pytest.mark.parametrize("lattice,dims", [(9, (64, 16, 1)), (27, (64, 16, 8))])
def test_infinities_and_nans_spread_as_in_fp64(cuda, lattice, dims):
    from cflbm import Solver
    E = E9 if lattice == 9 else E27
    nx, ny, nz = dims
    f = np.full((len(E), nz, ny, nx), 1e-3)
    f[1, 0, 4, 20], f[2, 0, 9, 40] = np.nan, np.inf
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.04, wall_y="periodic",
                wall_z="periodic", geom="none") as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
    g = np.stack([np.roll(f[i], e[::-1], (0, 1, 2)) for i, e in enumerate(E)])
    bad = ~np.isfinite(g).all(axis=0)
    ok = np.isfinite(got).all(axis=0)
    assert bad.sum() == 2 and (~ok == bad).all()


@pytest.mark.parametrize("lattice,dims", [(9, (67, 48, 1)), (27, (67, 32, 9))])
def test_one_step_error_with_porosity(cuda, lattice, dims):
    """Brinkman factors 1 - alpha inside [-1, 1] stay in the format (one more rounding,
    a quarter unit), others take FP64 operations."""
    from cflbm import Solver
    E = E9 if lattice == 9 else E27
    w = np.array([(np.longdouble(4) / 9 if lattice == 9 else np.longdouble(8) / 27)
                  / np.longdouble(4) ** sum(map(abs, e)) for e in E])
    nx, ny, nz = dims
    f = states(E, w, (nz, ny, nx))
    alpha = np.random.default_rng(6).choice([0.0, 0.3, 0.999, 1.0, 2.0, -0.5, 2.5], size=(nz, ny, nx))
    alpha = alpha.astype(np.float32).astype(np.float64)
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.03, u0=0.04, wall_y="periodic",
                wall_z="periodic", geom="none", alpha=alpha) as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
    ref, g = one_step(f, E, w, 1.0 / 0.53, np.longdouble(1) - alpha.astype(np.longdouble))
    ins = (slice(None), slice(None), slice(1, nx - 1))
    scale = np.abs(g / w.reshape(-1, 1, 1, 1)).max(axis=0)
    err = np.abs((got - ref) / w.reshape(-1, 1, 1, 1)).max(axis=0).astype(float)
    inside = (scale < 0.2 * (27 if lattice == 27 else 9)) & (np.abs(1 - alpha) <= 1)
    tol = np.where(inside, 13.0, 64.0 * (1.0 + 2.25 * scale)) * 2.0 ** -53 * scale
    tol = np.maximum(tol, 2.0 ** -940).astype(float)
    assert (err[ins] <= tol[ins]).all(), float((err[ins] / tol[ins]).max())
