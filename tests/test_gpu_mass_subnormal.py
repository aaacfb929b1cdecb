"""Domain sums of FP32 states with subnormal populations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,dims", [(9, (40, 9, 1)), (27, (33, 9, 5))])
def test_subnormal_populations_count(cuda, lattice, dims):
    from cflbm import Solver
    nx, ny, nz = dims
    with Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.02, u0=0.0, geom="none", storage="fp32",
                compute="fp32") as s:
        f = np.zeros((lattice, nz, ny, nx))
        f[1] = np.float32(1e-40)
        f[lattice - 1, :, :, ::3] = np.float32(-3e-42)
        s.set_f(f, steps_done=0)
        assert np.array_equal(s.get_f().reshape(f.shape), f)
        mom = s.mass()[1]
    from test_gpu_fixed_point import E9, E27
    E = np.array(E9 if lattice == 9 else E27, float)
    want = np.einsum("id,izyx->d", E, f)
    assert np.abs(mom - want).max() <= 1e-12 * np.abs(want).max()
