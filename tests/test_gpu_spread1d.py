"""1D spreading by register windows against the one-thread-per-point atomic kernel
(CUFINUFFT_KERNEL_VARIANT=1): sorted by cell and not, every method, counts around
the points-per-thread steps, points on one cell, wrapping windows, batches, both
precisions, both kernel forms, data outside FP32's range (FP64).  Bounds: FP32
rounding of sums in another order (2e-5, the parity bound), double-float (1e-13)."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single,tol,scale,kmeth", [(True, 1e-2, 1.0, 0), (True, 1e-6, 1.0, 0), (True, 1e-5, 1.0, 1),
                                                    (False, 1e-8, 1.0, 0), (False, 1e-10, 1e-200, 1),
                                                    (False, 1e-13, 1e100, 0)])
@pytest.mark.parametrize("N,M,kind", [(301, 1, "uniform"), (301, 3, "uniform"), (5000, 700, "uniform"),
                                      (301, 4001, "uniform"), (301, 4001, "onecell"), (64, 3000, "edge"),
                                      (2000, 155649, "series"), (2000, 622592, "uniform")])
def test_windows_against_atomics(monkeypatch, single, tol, scale, kmeth, N, M, kind):
    rng = np.random.default_rng(M)
    rdt, cdt = (np.float32, np.complex64) if single else (np.float64, np.complex128)
    if kind == "onecell":
        x = 0.5 + 1e-4 * rng.random(M)
    elif kind == "edge":
        x = np.pi * (1 - 0.02 * rng.random(M)) * rng.choice([-1, 1], M)
    elif kind == "series":
        x = (np.arange(M) + rng.random(M)) * (2 * np.pi / M) - np.pi
    else:
        x = rng.uniform(-np.pi, np.pi, M)
    ntr = 3 if M < 10000 else 1
    c = (NC.strengths(rng, M, ntr) * scale).astype(cdt)
    x = x.astype(rdt)
    kw = dict(ntr=ntr, maxbatchsize=2, gpu_kerevalmeth=kmeth)
    monkeypatch.setenv("CUFINUFFT_KERNEL_VARIANT", "1")
    ref, _ = NC.run_gpu(1, (N,), [x], c, tol, single, gpu_method=1, gpu_sort=0, **kw)
    monkeypatch.delenv("CUFINUFFT_KERNEL_VARIANT")
    # strengths of the sums, not the result: a crowded cell's terms may cancel
    size = np.linalg.norm(ref / scale)
    for m, sort in ((2, 1), (1, 1), (1, 0)):
        out, _ = NC.run_gpu(1, (N,), [x], c, tol, single, gpu_method=m, gpu_sort=sort, **kw)
        assert np.linalg.norm(out / scale - ref / scale) / size < (2e-5 if single else 1e-13), (m, sort)
