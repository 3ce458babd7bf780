"""1D type-1 points are sorted cell by cell only for the register-window kernels, which
share a cell's points: FP64 plans on FP64 instructions (tol below 1e-13, upsampfac below 2,
spreading alone) spread by atomics, which meet on one address in that order."""
import numpy as np
import pytest

from tests import nufft_cases as NC
from tests.launched import launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,tol,kw,by_cell", [
    (np.float32, 1e-5, {}, True), (np.float32, 1e-5, dict(gpu_method=1), False), (np.float64, 1e-9, {}, True), (np.float64, 1e-14, {}, False),
    (np.float64, 1e-9, dict(upsampfac=1.25), False), (np.float64, 1e-9, dict(gpu_spreadinterponly=1), False)])
def test_cell_sort_goes_with_the_windows(dt, tol, kw, by_cell):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(3)
    M = 60000
    x = torch.from_numpy(NC.points(rng, 1, M, dtype=dt, edges=False)[0]).cuda()
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64 if dt == np.float32 else np.complex128)).cuda()
    fk = torch.zeros(3000, dtype=c.dtype, device="cuda")
    plan = cufinufft(1, (3000,), eps=tol, dtype=dt, **kw)
    plan.set_pts(x)
    plan.execute(c, fk)
    assert ("k_scan_final" in launched(lambda: plan.set_pts(x))) == by_cell
    assert ("k_spread_win" in launched(lambda: plan.execute(c, fk))) == by_cell
