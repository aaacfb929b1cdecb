"""Dump, restore and domain sums over staging pieces, odd sizes and storages."""
import numpy as np
import pytest

from test_gpu_fixed_point import E9, E27

pytestmark = pytest.mark.gpu


def solver(lat, nx, ny, nz, storage, **kw):
    from cflbm import Solver
    return Solver(lattice=lat, nx=nx, ny=ny, nz=nz, storage=storage,
                  compute="fp64" if storage == "fp64" else "fp32", tau0=0.03, u0=0.05,
                  geom="cylinder", cx=nx / 3.0, cy=ny / 2.0, diam=ny / 3.0, perturb_amp=1e-3, **kw)


# the last: 70 MB, three staging pieces, and page mapping on several cores
@pytest.mark.parametrize("layout", ["rows", "soa"])
@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16dev"])
@pytest.mark.parametrize("shape", [(9, 5, 4, 1), (9, 130, 41, 1), (27, 33, 9, 7), (27, 161, 51, 40)])
def test_dump_and_restore(cuda, shape, storage, layout):
    lat, nx, ny, nz = shape
    rng = np.random.default_rng(2)
    w = 1e-3 * rng.normal(size=(lat, nz, ny, nx))
    store = {"fp64": np.float64, "fp32": np.float32, "fp16dev": None}[storage]
    with solver(*shape, storage, layout=layout) as s:
        s.set_f(w, steps_done=3)
        f = s.get_f().reshape(w.shape)
        assert s.info().steps_done == 3
        if store is not None:
            assert np.array_equal(f, w.astype(store).astype(np.float64))
        else:  # binary16 of the deviation from the free stream, half a unit at 2^-12 |f - b|
            assert np.abs(f - w).max() <= 2.0 ** -11 * 0.06
        s.set_f(f, steps_done=3)
        assert np.array_equal(s.get_f().reshape(w.shape), f)
        # mass and momentum: FP64 sums over the fluid cells in another order
        m, mom = s.mass()
        fluid = s.solid().reshape(nz, ny, nx) == 0
        E = np.array(E9 if lat == 9 else E27, float)
        g = f * fluid
        assert abs(m - (fluid.sum() + g.sum())) <= 1e-12 * fluid.sum()
        assert np.abs(mom - np.array([(E[:, d, None, None, None] * g).sum() for d in range(3)])).max() \
            <= 1e-12 * np.abs(g).sum()


def test_domain_sums_outside_the_integer_format(cuda):
    """Large populations take FP64 additions; a NaN is reported."""
    from cflbm import _lib as C
    with solver(27, 40, 12, 8, "fp64") as s:
        f = s.get_f()
        f[3, 2, 5, 7] = 1e3
        s.set_f(f)
        fluid = s.solid().reshape(8, 12, 40) == 0
        assert abs(s.mass()[0] - (fluid.sum() + (f * fluid).sum())) <= 1e-9
        f[3, 2, 5, 7] = np.nan
        s.set_f(f)
        with pytest.raises(Exception):
            s.mass()
