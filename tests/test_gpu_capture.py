"""A step captured by the caller: the force read before its first replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(lattice=9, nx=100, ny=40, tau0=0.03, u0=0.05, geom="cylinder", cx=25, cy=20, diam=8, perturb_amp=1e-3)


@pytest.mark.parametrize("storage,compute", [("fp64", "fp64"), ("fp32", "fp32")])
def test_force_of_captured_steps(cuda, storage, compute):
    """Captured launches write the history, not the slot of the last direct step: no
    force before the replay, each replay's own after it."""
    import torch
    from cflbm import Solver
    with Solver(**KW, storage=storage, compute=compute) as r, \
            Solver(**KW, storage=storage, compute=compute) as s:
        r.step(9)
        want = r.force_history()
        s.step(2)
        s.forces()
        s.step(1)
        assert np.array_equal(s.forces()[0], want[2])
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(s.stream_ptr())):
            g.capture_begin(capture_error_mode="thread_local")
            s.step(2)
            g.capture_end()
        assert not s.forces()[0].any()           # the history of steps that have not run
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.forces()[0], want[4])
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.forces()[0], want[4])  # step 5's entry, as before the replay
        s.step(2)                                # host count 7; device count 9
        assert np.array_equal(s.get_f(), r.get_f())
