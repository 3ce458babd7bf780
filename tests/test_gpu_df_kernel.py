"""The double-float kernel rows and tap sums of FP64 plans (exp form and
fitted polynomials) against the same plan on FP64 instructions
(CUFINUFFT_FP64_DF=0), over the kernel widths of tolerances 1e-7..1e-13 and
over data far outside FP32's exponent range.  Bound: 2^-46 per operation over
a few hundred sums in quadrature stays below 1e-13 relative l2."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmeth", [0, 1])
@pytest.mark.parametrize("dim,modes", [(2, (45, 38)), (3, (14, 17, 12))])
@pytest.mark.parametrize("tol,scale", [(9e-7, 1.0), (1e-7, 1e60), (1e-8, 1.0), (1e-10, 1.0), (1e-11, 1e-60),
                                       (1e-13, 1.0)])
def test_df_interp_against_fp64(monkeypatch, dim, modes, tol, scale, kmeth):
    rng = np.random.default_rng(int(-10 * np.log10(tol)) + dim)
    pts = NC.points(rng, dim, 3001, edges=False)
    fk = NC.coeffs(rng, modes) * scale
    kw = dict(gpu_method=2, gpu_kerevalmeth=kmeth)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    ref, _ = NC.run_gpu(2, modes, pts, fk, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF")
    out, info = NC.run_gpu(2, modes, pts, fk, tol, False, **kw)
    assert info["fp64_df"] == 1
    assert np.linalg.norm(out / scale - ref / scale) / np.linalg.norm(ref / scale) < 1e-13


@pytest.mark.parametrize("kmeth", [0, 1])
@pytest.mark.parametrize("M,sort", [(1, 1), (255, 0), (3001, 1), (19456, 1), (19457, 1)])
@pytest.mark.parametrize("tol,scale", [(9e-7, 1.0), (1e-7, 1e60), (1e-8, 1.0), (1e-10, 1e-250), (1e-12, 1.0),
                                       (1e-13, 1.0)])
def test_df_interp_1d(monkeypatch, M, sort, tol, scale, kmeth):
    rng = np.random.default_rng(M)
    pts = NC.points(rng, 1, M, lo=-3 * np.pi, hi=3 * np.pi, edges=False)
    fk = NC.coeffs(rng, (501,), 3) * scale
    kw = dict(gpu_kerevalmeth=kmeth, ntr=3, maxbatchsize=2, gpu_sort=sort)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    ref, _ = NC.run_gpu(2, (501,), pts, fk, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF")
    out, _ = NC.run_gpu(2, (501,), pts, fk, tol, False, **kw)
    assert np.linalg.norm(out / scale - ref / scale) / np.linalg.norm(ref / scale) < 1e-13


@pytest.mark.parametrize("kmeth", [0, 1])
@pytest.mark.parametrize("dim,modes,kw", [
    (2, (45, 38), dict(gpu_method=2)), (2, (64, 30), dict(gpu_method=3)),
    (2, (40, 40), dict(gpu_method=2, gpu_binsizex=7, gpu_binsizey=13, gpu_maxsubprobsize=33)),
    (3, (14, 17, 12), dict(gpu_method=2)), (3, (16, 12, 20), dict(gpu_method=4)),
    (3, (15, 15, 9), dict(gpu_method=2, gpu_binsizex=5, gpu_binsizey=3, gpu_binsizez=4, gpu_maxsubprobsize=31)),
    (3, (60, 10, 9), dict(gpu_method=2, gpu_binsizex=40, gpu_binsizey=2, gpu_binsizez=2))])
@pytest.mark.parametrize("tol,scale", [(9e-7, 1.0), (1e-7, 1e60), (1e-8, 1e-290), (1e-10, 1.0), (1e-11, 1e-60),
                                       (1e-12, 1.0), (1e-13, 1.0)])
def test_df_spread_against_fp64(monkeypatch, dim, modes, kw, tol, scale, kmeth):
    rng = np.random.default_rng(int(-10 * np.log10(tol)) + dim)
    pts = NC.points(rng, dim, 3001, edges=False)
    for p in pts:
        p[:1000] = p[0] + 1e-3 * rng.standard_normal(1000)   # a dense run
    c = NC.strengths(rng, 3001, 2) * scale
    kw = dict(kw, gpu_kerevalmeth=kmeth, ntr=2, maxbatchsize=2)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    ref, _ = NC.run_gpu(1, modes, pts, c, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF")
    out, _ = NC.run_gpu(1, modes, pts, c, tol, False, **kw)
    assert np.linalg.norm(out / scale - ref / scale) / np.linalg.norm(ref / scale) < 1e-13


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("dim,modes", [(2, (45, 38)), (3, (14, 17, 12))])
def test_df_zero_data(ntype, dim, modes):
    rng = np.random.default_rng(4)
    pts = NC.points(rng, dim, 700, edges=False)
    data = (NC.strengths(rng, 700) if ntype == 1 else NC.coeffs(rng, modes)) * 0.0
    out, _ = NC.run_gpu(ntype, modes, pts, data, 1e-9, False, gpu_method=2)
    assert not np.any(out)


@pytest.mark.parametrize("tol", [1e-1, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("dim,modes", [(2, (45, 38)), (3, (14, 17, 12))])
def test_df_narrow_kernels(monkeypatch, ntype, dim, modes, tol):
    """Widths 2..7, reached when FP64 plans keep FP64 throughout."""
    monkeypatch.setenv("CUFINUFFT_FP64_CHAIN", "1")
    rng = np.random.default_rng(dim)
    pts = NC.points(rng, dim, 3001, edges=False)
    data = NC.strengths(rng, 3001) if ntype == 1 else NC.coeffs(rng, modes)
    kw = dict(gpu_method=2)
    monkeypatch.setenv("CUFINUFFT_FP64_DF", "0")
    ref, _ = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF")
    out, _ = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw)
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 1e-13
