"""FP64 interpolation alone (gpu_spreadinterponly, type 2) of a grid that spans many
decades inside one tile: a point whose taps lie beside the large cells, not on them,
keeps the precision of its own taps.  Point by point against FP64 instructions
(CUFINUFFT_FP64_DF=0); bound: the two-sums of double-float rows keep ~2^-45 of a
point's own sum of a few hundred positive terms, 1e-12 with room."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmeth", [0, 1])
@pytest.mark.parametrize("large", [1e4, 1e8, 1e15])
@pytest.mark.parametrize("grid,M,method", [((240,), 3000, 1), ((64, 60), 40000, 1), ((64, 60), 40000, 2), ((64, 60), 40000, 0),
                                           ((36, 40, 32), 100000, 1), ((36, 40, 32), 100000, 2)])
@pytest.mark.parametrize("tol", [1e-7, 1e-10])
def test_beside_large_cells(monkeypatch, grid, M, method, large, kmeth, tol):
    rng = np.random.default_rng(M + len(grid))
    pts = NC.points(rng, len(grid), M, edges=False)
    fw = 1.0 + rng.random((1,) + grid[::-1]) + 1j * (1.0 + rng.random((1,) + grid[::-1]))
    spikes = fw.copy()
    spikes[(0,) + (slice(5, None, 24),) * len(grid)] = large
    kw = dict(gpu_spreadinterponly=1, gpu_method=method, gpu_kerevalmeth=kmeth)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    ref, _ = NC.run_gpu(2, grid, pts, spikes, tol, False, **kw)
    same, _ = NC.run_gpu(2, grid, pts, fw, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF")
    out, _ = NC.run_gpu(2, grid, pts, spikes, tol, False, **kw)
    beside = ref == same  # no tap on a large cell
    assert 0.2 < beside.mean() < 1.0
    rel = np.abs(out - ref) / np.abs(ref)
    assert rel[beside].max() < 1e-12, rel[beside].max()
