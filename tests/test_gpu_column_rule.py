"""Which 3D FP32 subproblems are spread by columns: on both sides of each line of the rule
(points of a column for narrow kernels, of the grid's cells and of a subproblem for the
others, the cell-run layout's own lines), the kernel by name and the result against
global atomics (1e-5: FP32 sums of up to ~1e4 terms in another order)."""
import numpy as np
import pytest

from tests import nufft_cases as NC
from tests.launched import launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol,density,method,bins,maxsub,columns", [
    (1e-4, 1.45, 2, (8, 8, 8), 1024, False), (1e-4, 1.55, 2, (8, 8, 8), 1024, True), (1e-4, 4.0, 2, (8, 8, 8), 256, False),
    (1e-3, 4.0, 2, (16, 16, 2), 1024, False), (1e-4, 3.9, 5, (8, 8, 8), 1024, False), (1e-4, 4.1, 5, (8, 8, 8), 1024, True),
    (1e-5, 0.39, 2, (8, 8, 8), 1024, False), (1e-5, 0.41, 2, (8, 8, 8), 1024, True), (1e-5, 1.0, 2, (16, 16, 2), 256, False),
    (1e-5, 2.1, 2, (16, 16, 2), 256, True), (1e-5, 2.0, 2, (8, 8, 4), 63, False), (1e-6, 0.9, 5, (8, 8, 8), 1024, False),
    (1e-6, 1.1, 5, (8, 8, 8), 1024, True)])
def test_kernel_and_result(tol, density, method, bins, maxsub, columns):
    import torch

    from cufinufft_gb300 import cufinufft
    modes = (24, 20, 18)
    rng = np.random.default_rng(int(100 * density))
    plan = cufinufft(1, modes[::-1], eps=tol, dtype=np.float32)
    i = plan.info()
    M = int(density * i["nf1"] * i["nf2"] * i["nf3"])
    plan.set_pts(*[torch.from_numpy(p).cuda() for p in NC.points(rng, 3, M, dtype=np.float32, edges=False)])
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64)).cuda()
    outs = []
    for m, b, ms in ((1, (16, 16, 2), 1024), (method, bins, maxsub)):
        plan.set_layout(m, b, ms)
        fk = torch.zeros(modes[::-1], dtype=c.dtype, device="cuda")
        names = launched(lambda: plan.execute(c, fk))
        outs.append(fk.cpu().numpy().astype(np.complex128))
    assert ("k_spread_sm_col" in names) == columns
    assert np.linalg.norm(outs[1] - outs[0]) / np.linalg.norm(outs[0]) < 1e-5
