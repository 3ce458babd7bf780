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
