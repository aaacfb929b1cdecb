"""The batch's one-launch step (blocks_per_sm = 0) against single channels: states and
fields bit for bit, forces to FP64 summation order (1e-12), for every tile height."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def configs(lattice, storage):
    out = []
    # odd sizes, a lone tile, no body, more than 512 boundary cells, walls of all kinds
    for k, (nx, ny, nz, d) in enumerate([(33, 9, 5, 3.0), (97, 30, 8, 9.0), (300, 260, 20, 200.0 if lattice == 9 else 9.0),
                                         (64, 12, 4, 0.0)]):
        if lattice == 27 and k == 2:
            nx, ny = 130, 40
        out.append(dict(lattice=lattice, nx=nx, ny=ny, nz=nz, tau0=0.03 + 0.01 * k, u0=0.05,
                        wall_y=("freeslip", "noslip", "periodic")[k % 3], wall_z=("periodic", "freeslip", "noslip")[k % 3],
                        geom="cylinder" if d else "none", cx=nx * 0.45, cy=ny / 2.0, diam=d,
                        perturb_amp=1e-3, seed=k, storage=storage, compute="fp32"))
    return out


@pytest.mark.parametrize("storage", ["fp32", "fp16dev", "fp64"])
@pytest.mark.parametrize("height", [1, 2, 4, 8])
@pytest.mark.parametrize("lattice", [9, 27])
def test_one_launch_step(cuda, lattice, height, storage):
    import torch
    from cflbm import Batch, Solver
    cfgs = configs(lattice, storage)
    with Batch(cfgs, graph_steps=4, autotune=False, tile_height=height, blocks_per_sm=0) as b:
        b.step(3)
        b.step(8)  # a captured graph and direct steps
        for k, cfg in enumerate(cfgs):
            s = b.instance(k)
            t = [torch.zeros(s.shape, dtype=torch.float64, device="cuda") for _ in range(4)]
            s.macros_device(*t)
            s.synchronize()
            with Solver(**cfg) as ref:
                ref.step(11)
                assert np.array_equal(s.get_f(), ref.get_f()), k
                for a, c, e in zip(t, s.macros(), ref.macros()):
                    assert np.array_equal(a.cpu().numpy(), e) and np.array_equal(c, e), k
                f, e = s.force_history(), ref.force_history()
                assert f.shape == e.shape == (11, 3)
                assert np.abs(f - e).max() <= 1e-12 * max(np.abs(e).max(), 1e-30), k
