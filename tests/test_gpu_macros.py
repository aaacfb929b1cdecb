"""Fields formed straight into a caller's device arrays against the handle's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [("fp64", "fp64"), ("fp64", "fp32"), ("fp32", "fp32"), ("fp32", "fp64"), ("fp16dev", "fp32"),
         ("fp16dev", "fp64")]
# partial last tiles, a lone last tile, whole pairs; body inside one tile and across tiles
SHAPES = [(9, 33, 21, 1), (9, 64, 16, 1), (9, 97, 30, 1), (27, 31, 9, 7), (27, 65, 12, 8), (27, 128, 16, 9)]


def channel(lattice, nx, ny, nz, storage, compute, wall):
    from cflbm import Solver
    return Solver(lattice=lattice, nx=nx, ny=ny, nz=nz, storage=storage, compute=compute, tau0=0.03,
                  u0=0.05, wall_y=wall, wall_z=wall, geom="cylinder", cx=nx / 3.0, cy=ny / 2.0,
                  diam=ny / 3.0, perturb_amp=1e-3, seed=3)


def device_fields(s, skip=()):
    import torch
    t = [None if k in skip else torch.full(s.shape, 7.0, dtype=torch.float64, device="cuda")
         for k in range(4)]
    s.macros_device(*t)
    s.synchronize()
    return [None if x is None else x.cpu().numpy() for x in t]


@pytest.mark.parametrize("storage,compute", FORMS)
@pytest.mark.parametrize("shape", SHAPES)
def test_direct_fields_equal_the_handles(cuda, shape, storage, compute):
    for wall in ("freeslip", "noslip", "periodic"):
        with channel(*shape, storage, compute, wall) as s:
            s.step(7)
            first = device_fields(s)            # formed in the caller's arrays
            partial = device_fields(s, (1, 2))  # formed in the handle, copied
            host = s.macros()
            f = s.get_f()
            s.set_f(f, steps_done=7)            # keeps the last step's fields
            after = s.macros()
        for k in range(4):
            assert np.array_equal(first[k], host[k]) and np.array_equal(after[k], host[k])
            assert partial[k] is None or np.array_equal(partial[k], host[k])
        # u and p of the step before, from its post-stream populations
        assert np.isfinite(first[0]).all() and np.abs(first[0]).max() < 1.0


@pytest.mark.parametrize("shape", [SHAPES[2], SHAPES[4]])
def test_partial_direct_request(cuda, shape):
    with channel(*shape, "fp32", "fp32", "noslip") as s:
        s.step(3)
        got = device_fields(s, (0, 2))          # first request, two arrays only
        host = s.macros()
    assert got[0] is None and np.array_equal(got[1], host[1]) and np.array_equal(got[3], host[3])


@pytest.mark.parametrize("storage,compute", FORMS)
@pytest.mark.parametrize("shape", SHAPES)
def test_fields_equal_post_stream_moments(cuda, shape, storage, compute):
    lat, nx, ny, nz = shape
    tol = 1e-12 if compute == "fp64" else 2e-6
    with channel(*shape, storage, compute, "noslip") as s:
        s.step(5)
        u, v, w, p = s.macros()
        g = s.get_f_stream().reshape((lat, nz, ny, nx))
        fluid = s.solid().reshape(nz, ny, nx) == 0
    rho3 = g.sum(axis=0)
    assert np.abs(p.reshape(rho3.shape) - rho3 / 3)[fluid].max() <= tol
    ex = [0, 1, 0, -1, 0, 1, -1, -1, 1] if lat == 9 else \
        [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1]
    ux = np.tensordot(np.array(ex, float), g, axes=1)
    assert np.abs(u.reshape(ux.shape) - ux)[fluid].max() <= tol
    assert np.abs(u.reshape(ux.shape))[~fluid].max(initial=0.0) == 0.0
