"""Default type-2 plans (method 1) whose points are dense enough run the tile
kernels: the result must equal the gather kernels' (set_layout with method 1
keeps those) up to the precision's rounding, on both sides of the density line,
for odd and given bins, batches, both precisions and the FP32 chain; plan info
stays that of method 1."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single,tol", [(True, 1e-5), (False, 1e-9), (False, 1e-6), (False, 1e-14)])
@pytest.mark.parametrize("modes,kw,per_bin", [
    ((50, 41), {}, (20, 101, 300)), ((33, 64), dict(gpu_binsizex=7, gpu_binsizey=13), (27, 130)),
    ((18, 13, 15), {}, (10, 60)), ((12, 14, 9), dict(gpu_binsizex=5, gpu_binsizey=3, gpu_binsizez=4), (47, 49)),
    ((40, 40), dict(gpu_maxsubprobsize=64), (200,)), ((64, 64), dict(gpu_binsizex=200, gpu_binsizey=200), (2000,)),
    ((40, 30), dict(gpu_sort=0), (200,))])
def test_routed_against_gather(single, tol, modes, kw, per_bin):
    import torch

    from cufinufft_gb300 import cufinufft
    rdt, cdt = (np.float32, np.complex64) if single else (np.float64, np.complex128)
    rng = np.random.default_rng(len(modes))
    fk = torch.from_numpy(NC.coeffs(rng, modes, 3, dtype=cdt)).cuda()
    plan = cufinufft(2, modes[::-1], n_trans=3, eps=tol, dtype=rdt, maxbatchsize=2, **kw)
    nb = plan.info()["nbins"]
    for n in per_bin:
        M = n * nb + 3
        pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, len(modes), M, lo=-3 * np.pi, hi=3 * np.pi, dtype=rdt,
                                                             edges=False)]
        outs = []
        for gather in (False, True):
            if gather:
                info = plan.info()
                assert info["method"] == 1 and info["nsubprob"] == 0
                ref_plan = cufinufft(2, modes[::-1], n_trans=3, eps=tol, dtype=rdt, maxbatchsize=2)
                ref_plan.set_pts(*pts[::-1])
                ref_plan.set_layout(1, (8,) * len(modes))
            p = ref_plan if gather else plan
            if not gather:
                p.set_pts(*pts[::-1])
            c = torch.zeros((3, M), dtype=fk.dtype, device="cuda")
            p.execute(c, fk)
            torch.cuda.synchronize()
            outs.append(c.cpu().numpy())
        diff = np.linalg.norm(outs[0] - outs[1]) / np.linalg.norm(outs[1])
        # the gather and tile kernels' own bounds: FP32 rounding of the rows and
        # sums (2e-5), double-float against FP64 (1e-13)
        assert diff < (2e-5 if single or tol >= 1e-6 else 1e-13), (n, diff)
