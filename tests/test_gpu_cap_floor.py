"""The route's subproblem cap: no smaller than an even bin's points where the bins fill the
chip, else by the points' number; the subproblems are those of the launch (block counts of
the profiler), the result that of the plan's own bins up to the order of FP32 sums."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


def _blocks(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile

    from tests.launched import launched
    launched(fn)  # (the process's first profile)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
        fn()
        torch.cuda.synchronize()
    import json
    import os
    import tempfile
    with tempfile.TemporaryDirectory() as d:
        prof.export_chrome_trace(os.path.join(d, "t.json"))
        ev = json.load(open(os.path.join(d, "t.json")))["traceEvents"]
    return [e["args"]["grid"][0] for e in ev if "k_spread_sm" in e.get("name", "") and "grid" in e.get("args", {})]


@pytest.mark.parametrize("modes,M,tol,bins,split", [
    ((300, 300), 90000, 1e-5, 19 * 19, False),       # 32^2 bins of 249 points, 361 of them
    ((250, 250), 62500, 1e-5, 16 * 16, True),        # 256 bins of 244
    ((32, 32, 32), 131072, 1e-5, 8 * 8 * 8, False),  # columns: 8^3 bins of 256
    ((32, 32, 32), 78643, 1e-5, 4 * 8 * 16, True),   # planes: 16x8x4 bins of 154, 512 of them
    ((48, 48, 48), 221184, 1e-5, 6 * 12 * 24, False)])
def test_even_bins(modes, M, tol, bins, split):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(M)
    plan = cufinufft(1, modes[::-1], eps=tol, dtype=np.float32)
    plan.set_pts(*[torch.from_numpy(p).cuda() for p in NC.points(rng, len(modes), M, dtype=np.float32, edges=False)])
    c = torch.from_numpy(NC.strengths(rng, M, dtype=np.complex64)).cuda()
    fk = torch.zeros(modes[::-1], dtype=c.dtype, device="cuda")
    blocks = _blocks(lambda: plan.execute(c, fk))
    assert len(blocks) == 1 and (blocks[0] > 1.5 * bins if split else blocks[0] <= 1.1 * bins), blocks
    out = fk.cpu().numpy().astype(np.complex128)
    plan.set_layout(2, (32, 32) if len(modes) == 2 else (16, 16, 2))
    plan.execute(c, fk)
    ref = fk.cpu().numpy().astype(np.complex128)
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 2e-5
