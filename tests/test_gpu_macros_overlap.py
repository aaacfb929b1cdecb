"""Fields requested into overlapping device arrays: as if copied u, v, w, p in turn."""
import numpy as np
import pytest

from test_gpu_macros import channel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,compute", [("fp64", "fp64"), ("fp32", "fp32")])
@pytest.mark.parametrize("starts", [(0, 0, 0, 0), (0, 1, 2, 3), (3, 2, 1, 0), (0, 700, None, 350)])
def test_overlapping_arrays(cuda, starts, storage, compute):
    import torch
    with channel(27, 65, 12, 8, storage, compute, "noslip") as s:
        s.step(3)
        n = s.nx * s.ny * s.nz
        buf = torch.full((n + 1000,), 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s.macros_device(*[None if o is None else buf[o:] for o in starts])
        s.synchronize()
        want = np.full(n + 1000, 7.0)
        for o, m in zip(starts, s.macros()):
            if o is not None:
                want[o:o + n] = np.asarray(m).ravel()
    assert np.array_equal(buf.cpu().numpy(), want)
