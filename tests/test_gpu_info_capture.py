"""Plan info is a query: inside a capture of the plan's stream, or beside one of
another thread, it gives what it gives outside and leaves the capture whole."""
import threading

import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other_thread", [False, True])
@pytest.mark.parametrize("ntype,modes,M,dt,tol", [
    (1, (50, 41), 30000, np.float32, 1e-5), (1, (18, 13, 15), 30000, np.float64, 1e-9),
    (1, (50, 41), 30000, np.float64, 1e-5), (1, (3000,), 40000, np.float32, 1e-5), (2, (50, 41), 30000, np.float32, 1e-5)])
def test_info_inside_a_capture(ntype, modes, M, dt, tol, other_thread):
    import torch

    from cufinufft_gb300 import cufinufft
    cdt = np.complex64 if dt == np.float32 else np.complex128
    rng = np.random.default_rng(M + len(modes))
    pts = NC.points(rng, len(modes), M, dtype=dt, edges=False)
    data = NC.strengths(rng, M, dtype=cdt) if ntype == 1 else NC.coeffs(rng, modes, dtype=cdt)
    ref, want = NC.run_gpu(ntype, modes, pts, data, tol, dt == np.float32)
    plan = cufinufft(ntype, modes[::-1], eps=tol, dtype=dt)
    s = torch.cuda.Stream()
    plan.set_stream(s.cuda_stream)
    d = torch.from_numpy(data).cuda()
    out = torch.zeros(modes[::-1] if ntype == 1 else (M,), dtype=d.dtype, device="cuda")
    dev = [torch.from_numpy(p).cuda() for p in pts]
    torch.cuda.synchronize()
    plan.set_pts(*dev[::-1])
    args = (d, out) if ntype == 1 else (out, d)
    plan.execute(*args)
    torch.cuda.synchronize()
    got = []

    def query():
        got.append(plan.info())

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        if other_thread:
            t = threading.Thread(target=query)
            t.start()
            t.join()
        else:
            query()
        plan.execute(*args)
    query()
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert got[0] == got[1] == want
    o = out.cpu().numpy()
    bound = 2e-5 if dt == np.float32 or tol >= 1e-6 else 1e-12
    assert np.linalg.norm(o - ref[0]) / np.linalg.norm(ref) < bound


def test_info_without_points():
    from cufinufft_gb300 import cufinufft
    for dt in (np.float32, np.float64):
        assert cufinufft(1, (40, 30), eps=1e-5, dtype=dt).info()["nsubprob"] == 0
