"""Large 3D FP32 point sets are sorted in two steps (positions, then copies): the
transform equals the unsorted one's, on both sides of the line, from coordinates
and for a new layout of points already sorted, cell-run layout included."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("M", [249999, 250000, 300001])
def test_sorted_against_unsorted(ntype, M):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(M)
    modes = (20, 18, 16)
    pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, 3, M, lo=-3 * np.pi, hi=3 * np.pi, dtype=np.float32,
                                                         edges=False)]
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64)).cuda()
    fk = torch.from_numpy(NC.coeffs(rng, modes, dtype=np.complex64)).cuda()

    def run(plan):
        c2, f2 = c.clone(), fk.clone()
        plan.execute(c2, f2)
        torch.cuda.synchronize()
        return (f2 if ntype == 1 else c2).cpu().numpy()

    ref = cufinufft(ntype, modes[::-1], eps=1e-5, dtype=np.float32, gpu_method=1, gpu_sort=0)
    ref.set_pts(*pts[::-1])
    want = run(ref)
    plan = cufinufft(ntype, modes[::-1], eps=1e-5, dtype=np.float32)
    plan.set_pts(*pts[::-1])
    got = [run(plan)]
    for layout in ((1, (8, 8, 8)), (2, (16, 8, 4))) + (((5, (8, 8, 8)),) if ntype == 1 else ()):
        plan.set_layout(*layout)
        got.append(run(plan))
    for out in got:
        # FP32 sums of up to ~1e3 terms in another order
        assert np.linalg.norm(out - want) / np.linalg.norm(want) < 2e-5
