"""Sorts whose points crowd few counters (blocks count in shared memory first), on both
sides of every line of that rule: the points from which it holds and from which a thread
takes more of them, one counter, the most counters and one bin more, points of the last
block; plain bins, bank classes and cells; points from coordinates, of an FP32 chain and
of a stored plan.  The transform against the unsorted one up to rounding, and the
subproblems' number against a host count."""
import numpy as np
import pytest

from tests import nufft_cases as NC
from tests.launched import launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,tol", [(np.float32, 1e-4), (np.float64, 1e-8), (np.float64, 1e-4)])
@pytest.mark.parametrize("ntype,modes,bins,M,crowded", [
    (1, (60, 60), (32, 32), 65535, False), (1, (60, 60), (32, 32), 65536, True), (1, (30, 30), (64, 64), 65543, True),
    (2, (60, 60), (32, 32), 70001, True), (2, (60, 60), (8, 8), 140000, False), (1, (60, 60), (2, 2), 461000, True),
    (1, (128, 128), (4, 4), 524288, True), (1, (128, 128), (4, 4), 524287, False), (1, (130, 128), (4, 4), 540800, False),
    (2, (20, 18, 16), (8, 8, 8), 220001, True), (1, (16, 16, 12), (16, 16, 2), 1245183, True),
    (1, (16, 16, 12), (16, 16, 2), 1245184, True), (1, (300,), (1024,), 80001, True), (2, (300,), (1024,), 80001, True),
    (1, (3000,), (1024,), 1300001, False)])
def test_sort_and_result(ntype, modes, bins, M, crowded, dt, tol):
    import torch

    from cufinufft_gb300 import cufinufft
    rdt, cdt = (torch.float32, torch.complex64) if dt == np.float32 else (torch.float64, torch.complex128)
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    dim = len(modes)
    pts = [(torch.rand(M, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * 3.1415 for _ in modes]
    for p in pts:
        p[M // 2:] = 0.3 + 0.2 * p[M // 2:]   # a crowded half
    pts = [p.to(rdt) for p in pts]
    n = modes[::-1]
    c = torch.randn(M, generator=g, device="cuda", dtype=cdt)
    fk = torch.randn(n, generator=g, device="cuda", dtype=cdt)
    kw = {"gpu_binsize" + "xyz"[k]: b for k, b in enumerate(bins)}
    if dim > 1 or ntype == 1:
        kw["gpu_method"] = 2
    outs = []
    for sort in (1, 0):
        plan = cufinufft(ntype, n, eps=tol, dtype=dt, **(kw if sort else dict(gpu_method=1, gpu_sort=0)))
        names = launched(lambda: plan.set_pts(*pts[::-1]))
        if sort:
            assert ("k_bin_count_crowded" in names) == crowded
        c2, f2 = c.clone(), fk.clone()
        plan.execute(c2, f2)
        outs.append((f2 if ntype == 1 else c2).to(torch.complex128))
        if sort and "gpu_method" in kw and dim > 1:   # the stored points once more, and back
            i = plan.info()
            plan.set_layout(1, bins)
            plan.set_layout(2, bins)
            assert plan.info()["nsubprob"] == i["nsubprob"]
            c2, f2 = c.clone(), fk.clone()
            plan.execute(c2, f2)
            outs.append((f2 if ntype == 1 else c2).to(torch.complex128))
    torch.cuda.synchronize()
    ref = outs.pop()
    # FP32 sums of up to 1e5 terms a cell in another order, double-float rows and sums
    bound = 2e-5 if dt == np.float32 or tol >= 1e-6 else 1e-12
    for out in outs:
        assert float((out - ref).norm() / ref.norm()) < bound
