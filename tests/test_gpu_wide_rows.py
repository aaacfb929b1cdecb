"""Rows so wide that a block's rows are more than 2^32 elements apart."""
import pytest

pytestmark = pytest.mark.gpu


def test_rows_beyond_32_bits(cuda):
    """FP64 arithmetic (one cell per thread, 32-bit offsets inside a block) against FP32
    (64-bit addresses) on one state, and their forces.  Both round every population to
    binary16 of its deviation d from the free stream, |d_i| <= 6 w_i u0 next to a wall
    or the body: after two such steps of two runs u is off by 4 x sum |e_i| 0.3 w_i 2^-11
    <= 2e-4, v likewise; rows differ by up to 1e-3 (the perturbation).
    """
    import torch
    from cflbm import Solver
    nx, ny = 160_000_000, 4
    kw = dict(lattice=9, nx=nx, ny=ny, tau0=0.05, u0=0.05, wall_y="noslip", geom="cylinder", cx=1.2e8,
              cy=2.0, diam=2.0, perturb_amp=1e-3, storage="fp16dev", rounding="nearest", force_history=4)
    fields, forces = [], []
    for compute in ("fp32", "fp64"):
        with Solver(**kw, compute=compute) as s:
            s.step(3)
            t = [torch.empty(s.shape, dtype=torch.float64, device="cuda") for _ in range(2)]
            s.macros_device(t[0], t[1], None, None)
            s.synchronize()
            forces.append(s.force_history(3))
            fields.append(t)
    for a, b in zip(*fields):
        assert float(a.std()) > 1e-4
        a -= b
        assert float(a.abs_().max()) <= 2e-4
    assert abs(forces[0] - forces[1]).max() <= 2e-4 * max(1.0, abs(forces[0]).max())
    del fields, t, a, b
    torch.cuda.empty_cache()
