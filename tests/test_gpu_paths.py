"""Each rule's path by kernel name, on both sides of the rule: double-float FFTs, spreads
and interpolations of FP64 plans and the FP64 forms, the tile route of default type-2
plans, the FP32 line FFT."""
import numpy as np
import pytest

from tests import nufft_cases as NC
from tests.launched import launched

pytestmark = pytest.mark.gpu


def _names(ntype, modes, M, dt, tol, **kw):
    import torch

    from cufinufft_gb300 import cufinufft
    cd = np.complex64 if dt == np.float32 else np.complex128
    rng = np.random.default_rng(M)
    plan = cufinufft(ntype, modes[::-1], eps=tol, dtype=dt, **kw)
    plan.set_pts(*[torch.from_numpy(p).cuda() for p in NC.points(rng, len(modes), M, dtype=dt, edges=False)][::-1])
    nt = kw.get("n_trans", 1)
    c = torch.from_numpy(NC.strengths(rng, M, nt, dtype=cd)).cuda()
    fk = torch.from_numpy(NC.coeffs(rng, modes, nt, dtype=cd)).cuda()
    return launched(lambda: plan.execute(c, fk))


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("modes,tol,passes", [
    ((1001,), 1e-9, 1), ((2048,), 1e-9, 1), ((20001,), 1e-11, 2), ((1001,), 1e-14, 0), ((50, 81), 1e-11, 2),
    ((64, 128), 1e-9, 2), ((9, 15, 27), 1e-9, 3), ((9, 15, 27), 1e-14, 0), ((50, 81), 1e-5, 0), ((2100, 10), 1e-9, 0)])
def test_df_fft(monkeypatch, ntype, modes, tol, passes):
    names = _names(ntype, modes, 3000, np.float64, tol)
    assert names.count("k_line_fft_df") == passes and ("fft" in names.replace("k_line_fft", "")) == (passes == 0)
    monkeypatch.setenv("CUFINUFFT_FP64_DF_FFT", "0")
    assert "k_line_fft_df" not in _names(ntype, modes, 3000, np.float64, tol)


@pytest.mark.parametrize("ntype,modes,M,tol,kw,kernel", [
    (2, (501,), 19456, 1e-9, {}, "k_interp_gm1_df_wide<"), (2, (501,), 19457, 1e-9, {}, "k_interp_gm1_df<"),
    (2, (501,), 3000, 1e-14, {}, "k_interp_gm_wc<"), (2, (501,), 3000, 1e-9, dict(upsampfac=1.25), "k_interp_gm_wc<"),
    (2, (45, 38), 30000, 1e-9, {}, "k_interp_sm_df<"), (2, (45, 38), 100, 1e-9, {}, "k_interp_gm_wc<"),
    (2, (45, 38), 300, 1e-9, dict(gpu_method=2), "k_interp_sm_df<"), (2, (45, 38), 30000, 1e-14, dict(gpu_method=2), "k_interp_sm<"),
    (2, (45, 38), 30000, 1e-14, {}, "k_interp_gm_wc<"), (2, (18, 17, 12), 30000, 1e-9, {}, "k_interp_sm_df<"),
    (1, (501,), 30000, 1e-9, {}, "k_spread_win_df<"), (1, (501,), 30000, 1e-14, {}, "k_spread_sm_wc<"),
    (1, (45, 38), 3000, 1e-9, {}, "k_spread_sm_priv_df<"), (1, (45, 38), 3000, 1e-14, {}, "k_spread_sm_priv<"),
    (1, (45, 38), 3000, 1e-9, dict(upsampfac=1.25), "k_spread_sm_priv<"),
    (1, (18, 17, 12), 3000, 1e-9, {}, "k_spread_sm_slab_df<"), (1, (18, 17, 12), 3000, 1e-14, {}, "k_spread_sm_wc<")])
def test_fp64_kernels(monkeypatch, ntype, modes, M, tol, kw, kernel):
    assert kernel in _names(ntype, modes, M, np.float64, tol, **kw)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    assert "_df" not in _names(ntype, modes, M, np.float64, tol, **kw)


@pytest.mark.parametrize("modes,M,kw,kernel", [
    ((100, 90), 3000, {}, "k_interp_gm_wc<"), ((100, 90), 30000, {}, "k_interp_sm<"),
    ((100, 90), 30000, dict(gpu_sort=0), "k_interp_gm_wc<"), ((24, 20, 18), 1000, {}, "k_interp_gm_wc<"),
    ((24, 20, 18), 50000, {}, "k_interp_sm<"), ((100, 90), 30000, dict(gpu_maxsubprobsize=64), "k_interp_gm_wc<")])
def test_fp32_tile_route(modes, M, kw, kernel):
    assert kernel in _names(2, modes, M, np.float32, 1e-5, **kw)


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("modes,line", [((512, 512), True), ((512, 511), True), ((256, 512), False), ((500, 600), False),
                                        ((128, 128, 128), True), ((64, 128, 64), False)])
def test_fp32_line_fft(ntype, modes, line):
    names = _names(ntype, modes, 3000, np.float32, 1e-5)
    assert ("k_line_fft_fx" in names) == line and names.count("k_line_fft") == (len(modes) if line else 0)


@pytest.mark.parametrize("M,kw,windows", [
    (30000, {}, True), (3000, {}, False), (30000, dict(gpu_method=1), False), (300000, dict(gpu_method=1), True),
    (30000, dict(gpu_method=0), False), (300000, dict(gpu_method=0), True)])
def test_fp32_1d_spread(M, kw, windows):
    assert ("k_spread_win<" in _names(1, (20001,), M, np.float32, 1e-5, **kw)) == windows


@pytest.mark.parametrize("M,nt,windows", [(100000, 1, True), (99999, 1, False), (200000, 4, True), (199999, 4, False)])
def test_sparse_1d_points(M, nt, windows):
    from cufinufft_gb300 import cufinufft
    assert cufinufft(1, (100000,), eps=1e-5, dtype=np.float32).info()["nf1"] == 200000
    kw = dict(gpu_method=2, n_trans=nt, maxbatchsize=nt)
    assert ("k_spread_win<" in _names(1, (100000,), M, np.float32, 1e-5, **kw)) == windows
