"""Crowded 1D FP32 cells: the grid that register windows spread is no further from 64 bits
than the tile kernel's shared atomics (CUFINUFFT_KERNEL_VARIANT=2) and than method 1 with
one thread per point (CUFINUFFT_KERNEL_VARIANT=1), whose sums meet one by one in the grid.
The grids themselves (spreading only), so that neither the kernel's nor the deconvolution's
error is in the way; the reference is the FP64 spread of the same width at the same points.
A block sums its windows before the grid, so its sums are no more than a tile's: its error
is at most theirs (a tenth more for what two orders of the same sums differ by)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,M", [(40, 200000), (600, 200000), (4000, 300000), (3750, 4000000), (200, 1000000)])
@pytest.mark.parametrize("tol", [1e-2, 1e-5])
def test_error_of_crowded_cells(monkeypatch, grid, M, tol):
    import torch

    from cufinufft_gb300 import cufinufft
    g = torch.Generator(device="cuda")
    g.manual_seed(grid)
    x = ((torch.rand(M, generator=g, device="cuda", dtype=torch.float64) * 2 - 1) * 3.1415).float()
    c = torch.randn(M, generator=g, device="cuda", dtype=torch.complex64)

    def spread(dt, cd, **kw):
        p = cufinufft(1, (grid,), eps=tol, dtype=dt, gpu_spreadinterponly=1, **kw)
        p.set_pts(x.to(torch.float32 if dt == np.float32 else torch.float64))
        fw = torch.zeros(grid, dtype=cd, device="cuda")
        p.execute(c.to(cd), fw)
        torch.cuda.synchronize()
        return fw.to(torch.complex128), p.info()["ns"]

    ref, ns = spread(np.float64, torch.complex128)
    windows, ns32 = spread(np.float32, torch.complex64)
    assert ns == ns32
    monkeypatch.setenv("CUFINUFFT_KERNEL_VARIANT", "2")
    tile, _ = spread(np.float32, torch.complex64, gpu_method=2)
    monkeypatch.setenv("CUFINUFFT_KERNEL_VARIANT", "1")
    points, _ = spread(np.float32, torch.complex64, gpu_method=1)
    err = [float((v - ref).norm() / ref.norm()) for v in (windows, tile, points)]
    print("grid %d M %d tol %g: windows %.2e, tile %.2e, one by one %.2e" % (grid, M, tol, *err))
    assert err[0] <= 1.1 * min(err[1:]) + 1e-9
