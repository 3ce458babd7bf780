"""1D FP32 spreading of thousands of points per cell: no further from 64 bits than
method 1 with one thread per point's own sums, on both sides of the span a block
sums in shared memory, and at the wrap of the grid."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes,M", [(40, 200000), (300, 200000), (2000, 200000), (16, 100), (1875, 4000000)])
@pytest.mark.parametrize("tol", [1e-2, 1e-5, 1e-7])
def test_error_against_double(modes, M, tol):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(modes)
    x = torch.from_numpy(rng.uniform(-np.pi, np.pi, M).astype(np.float32)).cuda()
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64)).cuda()
    out = []
    for dt, cd, eps in ((np.float32, torch.complex64, tol), (np.float64, torch.complex128, 1e-13)):
        p = cufinufft(1, (modes,), eps=eps, dtype=dt)
        p.set_pts(x.to(torch.float32 if dt == np.float32 else torch.float64))
        fk = torch.zeros(modes, dtype=cd, device="cuda")
        p.execute(c.to(cd), fk)
        torch.cuda.synchronize()
        out.append(fk.to(torch.complex128).cpu().numpy())
    err = np.linalg.norm(out[0] - out[1]) / np.linalg.norm(out[1])
    # the kernel's error, and FP32 coordinates, kernel values and sums: a few
    # 2^-24 per mode frequency up to modes / 2
    assert err < 10 * tol + 2e-6 * max(1.0, modes / 300), err
