"""setpts leaves nothing behind that still reads the caller's coordinates: when it
returns, the plan's stream is idle, the arrays may be overwritten on any stream, and
the plan may move to another stream; inside a caller's capture, where nothing runs
yet, a method-1 plan is recorded and can be used afterwards.  Results against plans
that set the same points undisturbed."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu

CASES = [  # type, modes, M, dtype, tol, options
    (1, (50, 41), 30000, np.float32, 1e-5, {}), (1, (50, 41), 30000, np.float64, 1e-9, {}),
    (1, (50, 41), 30000, np.float64, 1e-5, {}), (1, (18, 13, 15), 300000, np.float32, 1e-5, {}),
    (1, (3000,), 40000, np.float32, 1e-5, {}), (1, (50, 41), 30000, np.float32, 1e-5, dict(gpu_method=0)),
    (1, (50, 41), 30000, np.float32, 1e-5, dict(gpu_method=1)), (2, (50, 41), 30000, np.float32, 1e-5, {}),
    (2, (50, 41), 300, np.float32, 1e-5, {}), (2, (50, 41), 30000, np.float32, 1e-5, dict(gpu_sort=0)),
    (2, (18, 13, 15), 300000, np.float32, 1e-5, dict(gpu_method=2)), (2, (50, 41), 30000, np.float64, 1e-9, {}),
    (2, (3000,), 40000, np.float64, 1e-9, {})]


def _close(out, ref, dt, tol):
    bound = 2e-5 if dt == np.float32 or tol >= 1e-6 else 1e-12  # FP32 and double-float sums in another order
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < bound


def _setup(ntype, modes, M, dt, tol, opts):
    import torch

    from cufinufft_gb300 import cufinufft
    cdt = np.complex64 if dt == np.float32 else np.complex128
    rng = np.random.default_rng(M + ntype + len(modes))
    pts = NC.points(rng, len(modes), M, dtype=dt, edges=False)
    data = NC.strengths(rng, M, dtype=cdt) if ntype == 1 else NC.coeffs(rng, modes, dtype=cdt)
    ref, _ = NC.run_gpu(ntype, modes, pts, data, tol, dt == np.float32, **opts)
    plan = cufinufft(ntype, modes[::-1], eps=tol, dtype=dt, **opts)
    dev = [torch.from_numpy(p).cuda() for p in pts]
    d = torch.from_numpy(data).cuda()
    out = torch.zeros(modes[::-1] if ntype == 1 else (M,), dtype=d.dtype, device="cuda")
    torch.cuda.synchronize()
    return plan, dev, (d, out) if ntype == 1 else (out, d), out, ref[0]


@pytest.mark.parametrize("ntype,modes,M,dt,tol,opts", CASES)
def test_coordinates_overwritten_after_setpts(ntype, modes, M, dt, tol, opts):
    import torch
    plan, dev, args, out, ref = _setup(ntype, modes, M, dt, tol, opts)
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    plan.set_stream(own.cuda_stream)
    for _ in range(2):  # new plan arrays, then kept ones
        with torch.cuda.stream(own):
            torch.cuda._sleep(20_000_000)  # about 10 ms ahead of the sort
        keep = [p.clone() for p in dev]
        plan.set_pts(*dev[::-1])
        assert own.query(), "setpts returned with work left on the plan's stream"
        with torch.cuda.stream(other):
            for p in dev:
                p.uniform_(-3.0, 3.0)
        other.synchronize()
        out.zero_()
        torch.cuda.synchronize()
        plan.execute(*args)
        torch.cuda.synchronize()
        _close(out.cpu().numpy(), ref, dt, tol)
        for p, k in zip(dev, keep):
            p.copy_(k)
        torch.cuda.synchronize()


@pytest.mark.parametrize("ntype,modes,M,dt,tol,opts", CASES)
def test_stream_changed_after_setpts(ntype, modes, M, dt, tol, opts):
    import torch
    plan, dev, args, out, ref = _setup(ntype, modes, M, dt, tol, opts)
    plan.set_pts(*dev[::-1])
    s = torch.cuda.Stream()
    plan.set_stream(s.cuda_stream)
    plan.execute(*args)
    s.synchronize()
    _close(out.cpu().numpy(), ref, dt, tol)


@pytest.mark.parametrize("ntype,modes,M,dt,tol,opts", [c for c in CASES if c[0] == 2 and c[5].get("gpu_method", 1) == 1])
def test_setpts_recorded_in_a_graph(ntype, modes, M, dt, tol, opts):
    import torch
    plan, dev, args, out, ref = _setup(ntype, modes, M, dt, tol, opts)
    s = torch.cuda.Stream()
    plan.set_stream(s.cuda_stream)
    other = [torch.empty_like(p).uniform_(-3.0, 3.0) for p in dev]
    torch.cuda.synchronize()
    plan.set_pts(*other[::-1])
    plan.execute(*args)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.set_pts(*dev[::-1])
        plan.execute(*args)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    _close(out.cpu().numpy(), ref, dt, tol)
    assert plan.info()["nsubprob"] == 0
    for _ in range(3):  # direct, captured by the plan, replayed
        out.zero_()
        torch.cuda.synchronize()
        plan.execute(*args)
        s.synchronize()
        _close(out.cpu().numpy(), ref, dt, tol)
