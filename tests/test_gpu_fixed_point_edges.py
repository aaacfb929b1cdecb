"""Values at the edges of the block fixed-point format: what is not finite or far out
of it in any one population, exact zeros, an inlet value far above its cell's
populations, and slow relaxation.
"""
import numpy as np
import pytest

from test_gpu_fixed_point import E9, E27, one_step

pytestmark = pytest.mark.gpu

BAD = (np.nan, np.inf, -np.inf, 1e307)


def weights(lattice):
    E = E9 if lattice == 9 else E27
    return E, np.array([(np.longdouble(4) / 9 if lattice == 9 else np.longdouble(8) / 27)
                        / np.longdouble(4) ** sum(map(abs, e)) for e in E])


def pulled(f, E):
    return np.stack([np.roll(f[i], e[::-1], (0, 1, 2)) for i, e in enumerate(E)])


@pytest.mark.parametrize("storage,compute", [("fp64", "fp64"), ("fp64", "df64"), ("fp32", "fp64")])
@pytest.mark.parametrize("lattice,dims", [(9, (64, 16, 1)), (27, (64, 16, 8))])
def test_bad_value_in_any_one_population(cuda, lattice, dims, storage, compute):
    """Every (population, value) has a cell of its own; the same cells are finite as in
    FP64 arithmetic, populations and fields."""
    from cflbm import Solver
    E, w = weights(lattice)
    nx, ny, nz = dims
    f = np.full((len(E), nz, ny, nx), 1e-3)
    bad = BAD if storage == "fp64" else BAD[:3]
    for k, (i, v) in enumerate((i, v) for i in range(len(E)) for v in bad):
        e = E[i]
        x, y, z = 3 + 2 * (k % 28), 2 * (k // 28) + 1, k % nz
        f[i, (z - e[2]) % nz, (y - e[1]) % ny, x - e[0]] = v
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.04, wall_y="periodic",
                wall_z="periodic", geom="none", storage=storage, compute=compute) as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
        mac = [np.asarray(m).reshape(f.shape[1:]) for m in s.macros()]
    with np.errstate(all="ignore"):
        g = pulled(f, E)
        rho3 = g.sum(axis=0)
        u = [sum((e[d] * gi for e, gi in zip(E, g) if e[d]), np.zeros_like(rho3)) for d in range(3)]
        eu = [sum(e[d] * u[d] for d in range(3)) for e in E]
        usq = sum(c * c for c in u)
        feq = [float(wi) * (rho3 + 3 * a + 4.5 * a * a - 1.5 * usq) for wi, a in zip(w, eu)]
        ref = g - (g - np.stack(feq)) / 0.52
    ins = (Ellipsis, slice(1, nx - 1))
    assert (~np.isfinite(g)).any(axis=0).sum() == 3 * len(E)
    assert np.array_equal(np.isfinite(got)[ins], np.isfinite(ref)[ins])
    for m, r in zip(mac, u + [rho3 / 3]):
        assert np.array_equal(np.isfinite(m)[ins], np.isfinite(r)[ins])


@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16dev"])
@pytest.mark.parametrize("lattice,dims", [(9, (40, 9, 1)), (27, (40, 9, 5))])
def test_domain_sums_report_a_bad_value_in_any_population(cuda, lattice, dims, storage):
    from cflbm import Solver
    nx, ny, nz = dims
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.04, geom="none", storage=storage,
                compute="fp64" if storage == "fp64" else "fp32") as s:
        f0 = s.get_f().reshape((lattice, nz, ny, nx))
        for i in range(lattice):
            for v in BAD[:3]:
                f = f0.copy()
                f[i, nz // 2, 4, 21] = v
                s.set_f(f)
                with pytest.raises(Exception):
                    s.mass()
        s.set_f(f0)
        assert abs(s.mass()[0] - nx * ny * nz) < 1.0


@pytest.mark.parametrize("compute", ["fp64", "df64"])
@pytest.mark.parametrize("lattice,dims", [(9, (67, 20, 1)), (27, (67, 12, 9))])
def test_zeros_stay_zeros(cuda, lattice, dims, compute):
    """A fluid at rest and the inside of a body; and cells of zeros beside others."""
    from cflbm import Solver
    E, _ = weights(lattice)
    nx, ny, nz = dims
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.0, wall_y="noslip", wall_z="freeslip",
                geom="cylinder", cx=20, cy=ny / 2.0, diam=6, compute=compute) as s:
        f = np.zeros((lattice, nz, ny, nx))
        s.set_f(f, steps_done=0)
        s.step(3)
        assert not s.get_f().any() and not any(np.asarray(m).any() for m in s.macros())
    f = np.random.default_rng(3).normal(size=f.shape) * 1e-3
    f[..., ny // 2:, :] = 0.0
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.0, wall_y="periodic",
                wall_z="periodic", geom="none", compute=compute) as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
    empty = ~pulled(f, E).any(axis=0)
    assert empty.any() and not got[:, empty].any()


@pytest.mark.parametrize("u0", [0.05, 0.0625 * (1 - 2.0 ** -40), 3.0])
def test_inlet_value_far_above_its_cells(cuda, u0):
    """The reference profiles' inlet column over zero populations, solid cells in it
    included: omega feq(0, u_in).  16 roundings of the FP64 expression.  (Its end rows
    pull the corner ghosts, which this variant never writes.)"""
    from cflbm import Solver
    E, w = weights(9)
    w = w.astype(float)
    with Solver(lattice=9, nx=8, ny=65, profile="ref2ds", tau0=0.03, u0=u0) as s:
        assert s.solid().reshape(65, 8)[:, 0].any()
        s.set_f(np.zeros((9, 1, 65, 8)), steps_done=0)
        s.step(1)
        got = s.get_f().reshape((9, 65, 8))[:, 1:-1, 0]
        u = np.asarray(s.macros()[0]).reshape(65, 8)[1:-1, 0]
    y = np.arange(1.0, 64.0)
    uin = u0 * 4.0 * y * (64 - y) / 64.0 ** 2
    ref = np.stack([w[i] * (3 * e[0] * uin + 4.5 * (e[0] * uin) ** 2 - 1.5 * uin ** 2)
                    for i, e in enumerate(E)]) / 0.53
    assert np.abs(got - ref).max() <= 16 * 2.0 ** -53 * np.abs(ref).max()
    assert np.abs(u - uin).max() <= 4 * 2.0 ** -53 * u0


@pytest.mark.parametrize("tau0", [3.0, 100.0, 1e6])
@pytest.mark.parametrize("lattice,dims", [(9, (64, 20, 1)), (27, (64, 12, 5))])
def test_slow_relaxation_keeps_small_populations(cuda, lattice, dims, tau0):
    """At small omega a step moves a population by omega (feq - f): its error is a
    rounding or two of its own value and omega times the 64 of the FP64 equilibrium."""
    from cflbm import Solver
    E, w = weights(lattice)
    nx, ny, nz = dims
    rng = np.random.default_rng(8)
    f = 0.03 * rng.normal(size=(lattice, nz, ny, nx)) * w.reshape(-1, 1, 1, 1).astype(float)
    f *= 10.0 ** -rng.integers(0, 12, size=f.shape)
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=tau0, u0=0.04, wall_y="periodic",
                wall_z="periodic", geom="none") as s:
        s.set_f(f, steps_done=0)
        s.step(1)
        got = s.get_f().reshape(f.shape)
    omega = 1.0 / (tau0 + 0.5)
    ref, g = one_step(f, E, w, omega)
    w = w.reshape(-1, 1, 1, 1).astype(float)
    scale = w * np.abs(g / w).max(axis=0).astype(float)
    tol = 2.0 ** -53 * (2 * np.abs(g).astype(float) + 64 * omega * scale)
    assert (np.abs(got - ref).astype(float) <= tol)[..., 1:-1].all()


@pytest.mark.parametrize("compute", ["fp64", "df64"])
@pytest.mark.parametrize("wall_z", ["periodic", "freeslip"])
def test_spanwise_uniform_flow_stays_so(cuda, wall_z, compute):
    """Populations that mirror each other in z round alike, whichever pipe converts
    them: a flow uniform in z keeps w = 0 and equal layers, to the bit."""
    from cflbm import Solver
    with Solver(lattice=27, nx=90, ny=34, nz=9, tau0=0.0192, u0=0.05, wall_z=wall_z, geom="cylinder", cx=24,
                cy=15.3, diam=9, perturb_amp=0.0, compute=compute) as s:
        s.step(120)
        u, v, w, p = [np.asarray(m).reshape(9, 34, 90) for m in s.macros()]
        f = s.get_f().reshape(27, 9, 34, 90)
    assert np.abs(v).max() > 1e-3 and not w.any()
    for m in (u, v, p, *f):
        assert np.array_equal(m, np.broadcast_to(m[:1], m.shape))
