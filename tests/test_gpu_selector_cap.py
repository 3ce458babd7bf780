"""gpu_method 0, type 2, 4096 points a bin and 4096 * 1024 in all: whatever class the network
takes, full subproblems (their number is at most one more per bin than 1024 points each
need), and the result of the gather kernels up to FP32 rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes,M,eps,spread", [((33, 28, 32), 26000000, 1e-3, 0.05), ((33, 28, 32), 8000000, 1e-5, None),
                                                ((200, 180), 6000000, 1e-4, None)])
def test_full_subproblems(modes, M, eps, spread):
    import torch

    from cufinufft_gb300 import cufinufft
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    pts = []
    for _ in modes:
        x = (torch.rand(M, generator=g, device="cuda") * 2 - 1) * 3.1415
        if spread:
            x[M // 2:] = 0.4 + spread * torch.randn(M - M // 2, generator=g, device="cuda")
        pts.append(x)
    fk = torch.randn(modes, generator=g, device="cuda", dtype=torch.complex64)
    outs = []
    for method in (0, 1):
        plan = cufinufft(2, modes, eps=eps, dtype=np.float32, gpu_method=method)
        plan.set_pts(*pts)
        i = plan.info()
        c = torch.zeros(M, dtype=torch.complex64, device="cuda")
        if method == 1:
            plan.set_layout(1, (32,) * len(modes))
        plan.execute(c, fk)
        torch.cuda.synchronize()
        outs.append(c)
        if method == 0 and i["method"] == 2 and M >= 4096 * max(i["nbins"], 1024):
            assert i["nsubprob"] <= M // 1024 + i["nbins"], i
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 2e-5


@pytest.mark.parametrize("modes,M,sparse", [((438, 671), 1100000, True), ((323, 219), 274583, True), ((314, 515), 435715, True),
                                            ((239, 501), 142454, True), ((235, 296), 911085, True), ((180, 200), 150001, True),
                                            ((180, 200), 700000, False)])
def test_even_points_of_a_plan_among_others(modes, M, sparse):
    """2D FP32 type 2, uniform points: no 16^2 bins below four points per cell, and the bins
    that fill the chip are not split at 256 points."""
    import torch

    from cufinufft_gb300 import cufinufft
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    plan = cufinufft(2, modes, eps=1e-5, dtype=np.float32, gpu_method=0)
    plan.set_pts(*[(torch.rand(M, generator=g, device="cuda") * 2 - 1) * 3.1415 for _ in modes])
    i = plan.info()
    assert (M < 4 * i["nf1"] * i["nf2"]) == sparse
    if i["method"] == 2:
        assert not sparse or min(i["binsizex"], i["binsizey"]) >= 32, i
        assert i["nbins"] < 304 or i["nsubprob"] <= M // 1024 + i["nbins"], i
