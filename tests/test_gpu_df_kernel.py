"""The double-float kernel rows and tap sums of FP64 type-2 plans (exp form and
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
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 1e-13
