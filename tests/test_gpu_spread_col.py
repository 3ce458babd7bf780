"""3D FP32 spreading that sums the points of a column in registers (dense
subproblems, method 2 and the cell-run layout) against method 1 (global
atomics): every width, bins that leave one residue without a second plane, bins
deeper and shallower than the kernel, thin grids, subproblems longer than one
sort, crowded and even points, batches."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("tol", [10.0 ** -k for k in range(1, 8)])
@pytest.mark.parametrize("modes,bins,maxsub", [
    ((20, 18, 16), (8, 8, 8), 1024), ((20, 18, 16), (16, 8, 4), 37), ((9, 8, 30), (16, 16, 2), 1024),
    ((12, 12, 12), (5, 3, 13), 4096), ((14, 10, 12), (16, 16, 16), 3000), ((8, 7, 6), (1, 1, 40), 1024)])
def test_columns_against_global_atomics(crowded, tol, modes, bins, maxsub):
    rng = np.random.default_rng(len(bins) + maxsub)
    M = 16 * int(np.prod(modes))  # two points per grid cell
    pts = NC.points(rng, 3, M, lo=-3 * np.pi, hi=3 * np.pi, dtype=np.float32, edges=False)
    if crowded:
        for p in pts:
            p[: M // 2] = (0.3 + 0.02 * rng.standard_normal(M // 2)).astype(np.float32)
    c = np.stack([NC.strengths(rng, M, dtype=np.complex64) for _ in range(3)])
    import torch

    from cufinufft_gb300 import cufinufft
    plan = cufinufft(1, modes[::-1], n_trans=3, eps=tol, dtype=np.float32, maxbatchsize=2)
    plan.set_pts(*[torch.from_numpy(p).cuda() for p in pts[::-1]])
    cd = torch.from_numpy(c).cuda()
    outs = []
    for method, b in ((1, bins), (2, bins), (5, bins)):
        try:
            plan.set_layout(method, b, maxsub)
        except RuntimeError:
            assert method == 5  # no cell-run layout for some bins
            continue
        fk = torch.zeros((3,) + modes, dtype=cd.dtype, device="cuda")
        plan.execute(cd, fk)
        torch.cuda.synchronize()
        outs.append(fk.cpu().numpy())
    for out in outs[1:]:
        # FP32 sums of up to ~1e4 terms per cell in another order
        assert np.linalg.norm(out - outs[0]) / np.linalg.norm(outs[0]) < 1e-5


@pytest.mark.parametrize("tol", [10.0 ** -k for k in range(2, 8)])
@pytest.mark.parametrize("bins", [None, (8, 8, 8), (16, 8, 8)])
def test_wide_kernels(tol, bins):
    """Upsampling 1.25: widths up to 14, among them one whose block takes 48 KB of
    shared memory to the byte.  The grids themselves (spreading only): the
    deconvolution would amplify their rounding by orders of magnitude."""
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(5)
    grid = (36, 48, 40)
    M = 100000
    pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, 3, M, dtype=np.float32, edges=False)]
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64)).cuda()
    outs = []
    for method, b in ((1, (8, 8, 8)), (2, bins)):
        plan = cufinufft(1, grid[::-1], eps=tol, dtype=np.float32, upsampfac=1.25, gpu_spreadinterponly=1)
        plan.set_pts(*pts[::-1])
        if b:
            plan.set_layout(method, b)
        fk = torch.zeros(grid, dtype=c.dtype, device="cuda")
        plan.execute(c, fk)
        torch.cuda.synchronize()
        outs.append(fk.cpu().numpy().astype(np.complex128))  # squares leave FP32's range
    # FP32 sums of ns^3 taps of 1.4 points per cell in another order
    assert np.linalg.norm(outs[1] - outs[0]) / np.linalg.norm(outs[0]) < 1e-5
