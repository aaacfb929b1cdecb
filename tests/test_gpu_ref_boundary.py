"""The reference profiles' boundary launch against the sequential CPU restatement:
the passes' order at edges and corners, ghosts kept from step to step, links beside
the passes and, where the body comes within two cells of a face, after them.
Tolerance 1e-11: round-off of the FP64 steps."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def run(profile, nx, ny, nz, ran, steps, **kw):
    from cflbm import Solver
    with Solver(lattice=27 if profile == "ref3d" else 9, nx=nx, ny=ny, nz=nz, profile=profile,
                tau0=0.03, u0=0.04, ref_ran=ran, **kw) as s:
        for n in (1, 2, steps - 3):  # across calls as well
            s.step(n)
        u, v, w, p = s.macros()
        return dict(u=u, v=v, w=w, p=p, fpost=s.get_f(), force=s.force_history())


@pytest.mark.parametrize("layout", ["rows", "soa"])
@pytest.mark.parametrize("profile,nx,ny", [("ref2d", 12, 9), ("ref2d", 97, 4), ("ref2d", 130, 33),
                                           ("ref2d", 300, 6), ("ref2ds", 40, 17), ("ref2ds", 131, 34)])
def test_2d(cuda, profile, nx, ny, layout):
    ran = np.random.default_rng(3).integers(0, 100, size=(nx + 4, ny + 4)).astype(np.int32)
    o = (O.ref2d if profile == "ref2d" else O.ref2ds)(nx, ny, 0.03, 0.04, ran, 70)
    r = run(profile, nx, ny, 1, ran, 70, layout=layout)
    sl = (slice(2, 2 + nx), slice(2, 2 + ny))
    for k in ("u", "v", "p"):
        assert rel_err(r[k].reshape(ny, nx), o[k][sl].T) < 1e-11, k
    assert rel_err(r["fpost"].reshape(9, ny, nx), o["fpost"][(slice(None),) + sl].transpose(0, 2, 1)) < 1e-11
    if profile == "ref2d":
        assert rel_err(r["force"][:, :2], o["force"]) < 1e-9


@pytest.mark.parametrize("layout", ["rows", "soa"])
@pytest.mark.parametrize("nx,ny,nz", [(10, 9, 8), (17, 11, 9), (33, 8, 13), (70, 20, 12)])
def test_3d(cuda, nx, ny, nz, layout):
    ran = np.random.default_rng(3).integers(0, 100, size=(nx + 6, ny + 6, nz + 6)).astype(np.int32)
    o = O.ref3d(nx, ny, nz, 0.03, 0.04, ran, 70)
    r = run("ref3d", nx, ny, nz, ran, 70, layout=layout)
    sl = (slice(3, 3 + nx), slice(3, 3 + ny), slice(3, 3 + nz))
    for k in ("u", "v", "w", "p"):
        assert rel_err(r[k].reshape(nz, ny, nx), o[k][sl].transpose(2, 1, 0)) < 1e-11, k
    assert rel_err(r["fpost"].reshape(27, nz, ny, nx),
                   o["fpost"][(slice(None),) + sl].transpose(0, 3, 2, 1)) < 1e-11
