"""Default type-1 plans sort by the route's own bins and subproblem cap: the result
must equal the plan's own bins' (set_layout keeps those) up to the order of the
sums, for even and crowded points, on both sides of every line of the rule, and
plan info stays that of the plan's own layout."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("single,tol", [(True, 1e-2), (True, 1e-5), (True, 1e-7), (False, 1e-6), (False, 1e-10),
                                        (False, 1e-12), (False, 1e-13), (False, 1e-15)])
@pytest.mark.parametrize("modes,counts", [((50, 41), (1, 300, 30000)), ((9, 120), (900, 20000)),
                                          ((18, 13, 15), (2, 3000, 40000)), ((40, 7, 6), (5000,))])
def test_against_own_bins(crowded, single, tol, modes, counts):
    import torch

    from cufinufft_gb300 import cufinufft
    rdt, cdt = (np.float32, np.complex64) if single else (np.float64, np.complex128)
    if len(modes) == 3 and tol < 1e-14:
        pytest.skip("width 16: the default 16x16x2 tile does not fit, before and after")
    rng = np.random.default_rng(len(modes))
    plan = cufinufft(1, modes[::-1], n_trans=3, eps=tol, dtype=rdt, maxbatchsize=2)
    own = cufinufft(1, modes[::-1], n_trans=3, eps=tol, dtype=rdt, maxbatchsize=2)
    for M in counts:
        pts = NC.points(rng, len(modes), M, lo=-3 * np.pi, hi=3 * np.pi, dtype=rdt, edges=False)
        if crowded:
            for p in pts:
                p[: M // 2] = (0.3 + 0.01 * rng.standard_normal(M // 2)).astype(rdt)
        c = torch.from_numpy(np.stack([NC.strengths(rng, M, dtype=cdt) for _ in range(3)])).cuda()
        outs, infos = [], []
        for q in (plan, own):
            q.set_pts(*[torch.from_numpy(p).cuda() for p in pts[::-1]])
            if q is own:
                i = q.info()
                q.set_layout(i["method"], tuple(i["binsize" + "xyz"[k]] for k in range(len(modes))))
            fk = torch.zeros((3,) + modes, dtype=c.dtype, device="cuda")
            q.execute(c, fk)
            torch.cuda.synchronize()
            outs.append(fk.cpu().numpy())
            infos.append(q.info())
        for key in ("method", "binsizex", "binsizey", "binsizez", "nbins", "nsubprob"):
            assert infos[0][key] == infos[1][key], key
        diff = np.linalg.norm(outs[0] - outs[1]) / np.linalg.norm(outs[1])
        # sums of up to 4e4 terms in another order: FP32 2e-5 (also an FP64 plan from
        # tol 1e-6, which runs an FP32 chain); double-float rows and sums 1e-12
        assert diff < (2e-5 if single or tol >= 1e-6 else 1e-12), (M, diff)
