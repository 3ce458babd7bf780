"""gpu_method 0: the network, trained on single transforms, takes the layout from the
points alone, whatever the number of transforms that share them."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("modes,M,dt,tol", [
    ((45, 38), 30000, np.float32, 1e-5), ((300, 256), 500000, np.float32, 1e-3), ((45, 38), 30000, np.float64, 1e-9),
    ((64, 60, 50), 400000, np.float32, 1e-3), ((32, 30, 28), 100000, np.float64, 1e-9), ((5003,), 400000, np.float32, 1e-4)])
def test_layout_of_many_transforms(ntype, modes, M, dt, tol):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(M)
    pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, len(modes), M, dtype=dt, edges=False)][::-1]
    got = []
    for nt in (1, 3, 64):
        plan = cufinufft(ntype, modes[::-1], n_trans=nt, eps=tol, dtype=dt, gpu_method=0, maxbatchsize=1)
        plan.set_pts(*pts)
        i = plan.info()
        got.append([i[k] for k in ("method", "binsizex", "binsizey", "binsizez", "nsubprob")])
    assert got[0] == got[1] == got[2]
