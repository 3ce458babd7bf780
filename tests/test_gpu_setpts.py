"""The sort of set_pts: bin counters (sector-strided, plain, by bank class), the
one-pass scan over one and several blocks, headers written to their upper
bound, and repeated calls without a wait between them.  The subproblem count
must equal a host count of the bins, and the transform the unsorted one's up to
FP32 rounding (2e-5, the parity bound of FP32 kernels)."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


def _host_nsub(info, pts, maxsub):
    b = np.zeros(pts[0].size, dtype=np.int64)
    mul = 1
    for k, p in enumerate(pts):
        nf = info[f"nf{k + 1}"]
        bs = info["binsize" + "xyz"[k]]
        t = (p.astype(np.float64) / (2 * np.pi) + 0.5) * nf
        i0 = np.ceil(t - info["ns"] / 2).astype(np.int64) % nf
        b += mul * (i0 // bs)
        mul *= (nf + bs - 1) // bs
    c = np.bincount(b)
    return int(np.sum((c + maxsub - 1) // maxsub))


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("modes,bins,maxsub,M", [
    ((64, 48), (32, 32), 1024, 1), ((64, 48), (32, 32), 1024, 256), ((64, 48), (32, 32), 7, 257),
    ((300, 256), (4, 4), 64, 30000),      # 20k bins: five scan blocks, plain counters
    ((90, 90), (2, 1), 16, 5000),         # 16.2k bins
    ((256, 32), (8, 1), 16, 40000),       # 4096 bins: one scan block exactly
    ((257, 32), (8, 1), 16, 40000),       # two
    ((20, 18, 16), (16, 16, 2), 33, 4000), ((20, 18, 16), (3, 5, 7), 1024, 4000)])
def test_sort_counts_and_result(ntype, modes, bins, maxsub, M):
    rng = np.random.default_rng(M + len(modes))
    pts = NC.points(rng, len(modes), M, dtype=np.float32, edges=False)
    if M > 1000:   # a crowded corner: several subproblems of one bin
        for p in pts:
            p[: M // 2] = (0.3 + 0.01 * rng.standard_normal(M // 2)).astype(np.float32)
    data = NC.strengths(rng, M, dtype=np.complex64) if ntype == 1 else NC.coeffs(rng, modes, dtype=np.complex64)
    kw = {"gpu_binsize" + "xyz"[k]: b for k, b in enumerate(bins)}
    out, info = NC.run_gpu(ntype, modes, pts, data, 1e-4, True, gpu_method=2, gpu_maxsubprobsize=maxsub, **kw)
    ref, _ = NC.run_gpu(ntype, modes, pts, data, 1e-4, True, gpu_method=1, gpu_sort=0)
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 2e-5
    host = _host_nsub(info, pts, maxsub)
    # a point within FP32 rounding of a cell edge may fall on either side
    assert abs(info["nsubprob"] - host) <= 0.002 * host + 1


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("method", [0, 2])
def test_moving_points_without_waits(single, method):
    """set_pts / execute in a row with other point counts, nothing waited for."""
    import torch

    from cufinufft_gb300 import cufinufft
    rdt, cdt = (np.float32, np.complex64) if single else (np.float64, np.complex128)
    rng = np.random.default_rng(8)
    modes = (60, 44)
    plan = cufinufft(1, modes[::-1], eps=1e-5, dtype=rdt, gpu_method=method)
    jobs = []
    for M in (5000, 17, 20000, 800, 20000):
        pts = NC.points(rng, 2, M, dtype=rdt, edges=False)
        c = NC.strengths(rng, M, dtype=cdt)
        dev = [torch.from_numpy(p).cuda() for p in pts]
        jobs.append((pts, c, dev, torch.from_numpy(c).cuda(), torch.zeros(modes[::-1], dtype=getattr(torch, cdt.__name__), device="cuda")))
    torch.cuda.synchronize()
    for _, _, dev, c, fk in jobs:
        plan.set_pts(*dev[::-1])
        for _ in range(3):   # direct, captured, replayed
            plan.execute(c, fk)
    torch.cuda.synchronize()
    for pts, c, _, _, fk in jobs:
        ref, _ = NC.run_gpu(1, modes, pts, c, 1e-5, single, gpu_method=1, gpu_sort=0)
        assert np.linalg.norm(fk.cpu().numpy() - ref[0]) / np.linalg.norm(ref) < 2e-5
