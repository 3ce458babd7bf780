"""Bins whose FP64 tile all but fills a block's shared memory (232448 bytes): the
double-float kernels' static tables do not fit beside it, the FP64 kernels' few bytes
do, so such calls run -- against the default bins' result, in double-float: 1e-12."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


def _against_default_bins(ntype, modes, bins, tol, ns):
    rng = np.random.default_rng(sum(bins))
    M = 6000
    pts = NC.points(rng, len(modes), M, lo=-3 * np.pi, hi=3 * np.pi, edges=False)
    data = NC.strengths(rng, M, 2) if ntype == 1 else NC.coeffs(rng, modes, 2)
    kw = dict(ntr=2, maxbatchsize=2, gpu_method=2)
    ref, _ = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw)
    out, info = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw,
                           **{"gpu_binsize" + "xyz"[k]: b for k, b in enumerate(bins)})
    assert info["ns"] == ns and tuple(info["binsize" + "xyz"[k]] for k in range(len(bins))) == bins
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 1e-12


@pytest.mark.parametrize("bins,tol,ns", [((66, 24), 1e-10, 11), ((80, 24), 1e-10, 11), ((50, 29), 1e-11, 12),
                                         ((18, 51), 1e-13, 14), ((33, 51), 1e-13, 14), ((66, 23), 1e-10, 11)])
def test_spread_private_tiles(bins, tol, ns):
    _against_default_bins(1, (60, 44), bins, tol, ns)


@pytest.mark.parametrize("modes,bins,tol,ns", [((20, 34, 20), (13, 26, 15), 1e-7, 8), ((20, 20, 34), (13, 15, 26), 1e-7, 8),
                                               ((20, 24, 28), (13, 18, 22), 1e-7, 8), ((20, 24, 28), (13, 18, 21), 1e-7, 8)])
def test_interpolation_tiles(bins, modes, tol, ns):
    _against_default_bins(2, modes, bins, tol, ns)


def test_refused_call_leaves_no_error_behind():
    """Bins that leave the FP64 kernel's own few static bytes no room are refused by the
    launch; plans made and run after that are not."""
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(0)
    pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, 2, 6000, edges=False)]
    c = torch.from_numpy(NC.strengths(rng, 6000)).cuda()
    fk = torch.zeros((70, 60), dtype=c.dtype, device="cuda")
    refused = cufinufft(1, (70, 60), eps=1e-10, dtype=np.float64, gpu_method=2, gpu_binsizex=18, gpu_binsizey=62)
    refused.set_pts(*pts[::-1])
    for dt, modes in ((np.float64, (70, 60)), (np.float64, (3000,)), (np.float32, (512, 512)), (np.float64, (12, 14, 15))):
        with pytest.raises(RuntimeError):
            refused.execute(c, fk)
        plan = cufinufft(1, modes, eps=1e-10 if dt == np.float64 else 1e-5, dtype=dt)
        x = [pts[0].to(torch.float64 if dt == np.float64 else torch.float32)] * len(modes)
        plan.set_pts(*x)
        v = c if dt == np.float64 else c.to(torch.complex64)
        plan.execute(v, torch.zeros(modes, dtype=v.dtype, device="cuda"))
        torch.cuda.synchronize()
