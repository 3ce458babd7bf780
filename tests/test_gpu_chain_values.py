"""FP64 type-2 plans at tol >= 1e-6 run an FP32 chain whose sums show in the low bits of
their complex128 values: such a plan keeps one kernel and one FFT whatever the density
and the grid.  Dense default plans against the gather kernel and cuFFT by name
(CUFINUFFT_KERNEL_VARIANT=2, CUFINUFFT_FFT=cufft): the same kernels on the same inputs,
nothing random in type 2, so the values are equal.  With gpu_method 0 the layout is the
one that the chain's own network predicts."""
import os

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("tol", [1e-6, 1e-3])
@pytest.mark.parametrize("modes,M", [((50, 41), 20000), ((512, 512), 30000), ((320, 321), 201603), ((2047, 128), 400000),
                                     ((18, 13, 15), 30000), ((64, 60, 50), 700000), ((128, 128, 128), 20000)])
def test_default_plan_keeps_its_sums(monkeypatch, modes, M, tol):
    rng = np.random.default_rng(M + len(modes))
    pts = NC.points(rng, len(modes), M, edges=False)
    fk = NC.coeffs(rng, modes, 3)
    kw = dict(ntr=3, maxbatchsize=2)
    out, info = NC.run_gpu(2, modes, pts, fk, tol, False, **kw)
    assert info["chain_fp32"] == 1 and info["line_fft"] == 0
    monkeypatch.setenv("CUFINUFFT_KERNEL_VARIANT", "2")
    monkeypatch.setenv("CUFINUFFT_FFT", "cufft")
    ref, _ = NC.run_gpu(2, modes, pts, fk, tol, False, **kw)
    assert np.array_equal(out, ref), np.linalg.norm(out - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("modes,M,tol,sigma", [((353, 80, 79), 374087, 1e-3, 0.9), ((2324, 683), 121194, 1e-6, None),
                                               ((269, 250), 97303, 1e-3, 0.024), ((160, 479), 96795, 1e-3, 0.03),
                                               ((64, 60, 50), 700000, 1e-6, None)])
def test_layout_by_the_chains_network(modes, M, tol, sigma):
    import torch

    from cufinufft_gb300 import cufinufft
    _, mu, sd, params = MO.read_weights_header(os.path.join(ROOT, "cufinufft_gb300", "csrc", "selector_weights_chain.h"))
    rng = np.random.default_rng(M)
    pts = NC.points(rng, len(modes), M, edges=False)
    if sigma:
        for p in pts:
            p[:] = np.clip(0.7 + sigma * rng.standard_normal(M), -3.1, 3.1)
    plan = cufinufft(2, modes[::-1], eps=tol, dtype=np.float64, gpu_method=0)
    plan.set_pts(*[torch.from_numpy(p).cuda() for p in pts[::-1]])
    f, info = plan.features(), plan.info()
    assert info["chain_fp32"] == 1
    Y = MO.forward(params, ((f - mu) / sd)[None, :])[0][0]
    keys = ("method", "binsizex", "binsizey", "binsizez")
    runnable = {}
    for k in range(MO.K):
        try:
            plan.set_layout_class(k)
        except RuntimeError:
            continue
        runnable[k] = tuple(plan.info()[key] for key in keys)
    best = min(Y[k] for k in runnable)
    # FP32 against FP64 sums of the network: near-ties accept either
    assert tuple(info[key] for key in keys) in [v for k, v in runnable.items() if Y[k] <= best + 1e-3]
