"""The body force formed in the sweep's launch against the momentum exchange summed
on the host from the state the step reads.

Tolerances, relative to the sum of the terms' magnitudes: FP64 1e-13 (the order of
at most 2e5 additions), FP32 collision 1e-6 (per-cell sums of at most 26 terms in
FP32, exact from there).
"""
import numpy as np
import pytest

from test_gpu_fixed_point import E9, E27

pytestmark = pytest.mark.gpu


def exchange(f, solid, E):
    """(force, sum of magnitudes) of state f [Q, nz, ny, nx]; the body is inside."""
    F, mag = np.zeros(3), 0.0
    for e in E[1:]:
        src = np.roll(solid, e[::-1], (0, 1, 2))          # solid at X - e
        m = 2.0 * f[E.index(tuple(-v for v in e))][src & ~solid]
        F -= np.array(e) * m.sum()
        mag += np.abs(m).sum()
    return F, mag


# boundary cells: none, one block (<= 128, <= 512), several blocks, more than the SMs hold
CASES = [(9, 64, 33, 1, "none", 0.0), (9, 67, 40, 1, "cylinder", 9.0), (9, 500, 300, 1, "cylinder", 120.0),
         (9, 900, 700, 1, "cylinder", 500.0), (27, 48, 30, 24, "sphere", 9.0),
         (27, 96, 48, 90, "cylinder", 30.0)]


@pytest.mark.parametrize("storage,compute,tol", [("fp64", "fp64", 1e-13), ("fp64", "fp32", 1e-6),
                                                 ("fp32", "fp32", 1e-6), ("fp16dev", "fp32", 1e-6)])
@pytest.mark.parametrize("case", CASES)
def test_force_is_the_momentum_exchange(cuda, case, storage, compute, tol):
    from cflbm import Solver
    lat, nx, ny, nz, geom, d = case
    with Solver(lattice=lat, nx=nx, ny=ny, nz=nz, tau0=0.03, u0=0.05, wall_y="freeslip", geom=geom,
                cx=nx * 0.4, cy=ny / 2.0, cz=nz / 2.0, diam=d, perturb_amp=1e-3, storage=storage,
                compute=compute) as s:
        E = E9 if lat == 9 else E27
        solid = s.solid().reshape(nz, ny, nx).astype(bool)
        for n in (1, 2):
            s.step(n)
            f = s.get_f().reshape((lat, nz, ny, nx))
            s.step(1)
            F, mag = exchange(f, solid, E)
            assert np.abs(s.force_history(1)[-1] - F).max() <= tol * max(mag, 1e-300)
        assert s.force_history().shape == (5, 3)


def test_force_where_the_grid_is_full(cuda):
    """ny at the launch limit: the same force as in a box with room for its blocks
    (the far wall is out of the body's reach)."""
    from cflbm import Solver
    out = []
    for ny in (65535 * 4, 65000 * 4):
        with Solver(lattice=9, nx=24, ny=ny, tau0=0.03, u0=0.05, geom="cylinder", cx=10, cy=40,
                    diam=8, perturb_amp=1e-3, storage="fp32", compute="fp32") as s:
            s.step(5)
            out.append(s.force_history())
    assert np.array_equal(out[0], out[1])
