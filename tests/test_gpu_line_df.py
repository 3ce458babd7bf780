"""Double-float line FFTs of FP64 plans (fft_df.cu) against cuFFT's Z2Z
(CUFINUFFT_FP64_DF_FFT=0): 1D to 3D, lengths of every radix, one-pass lengths,
the longest line and the two-pass 1D form, odd mode counts, both signs, partial
batches, data outside FP32's range.  Bound: ~2^-46 per operation over a few dozen
butterfly levels stays below 1e-13 relative l2."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("modes,tol,iflag,ntr,scale", [
    ((7,), 1e-9, 1, 1, 1.0), ((1001,), 1e-9, -1, 3, 1.0), ((2047,), 1e-12, 1, 1, 1e-100),
    ((2048,), 1e-9, 1, 1, 1.0), ((2100,), 1e-10, -1, 2, 1e100), ((20001,), 1e-11, 1, 3, 1.0),
    ((65536,), 1e-12, -1, 1, 1.0),
    ((9, 12), 1e-7, 1, 1, 1.0), ((50, 81), 1e-11, -1, 5, 1.0), ((1500, 11), 1e-9, 1, 1, 1e-60),
    ((75, 240), 1e-12, 1, 2, 1.0), ((64, 2000), 1e-9, -1, 1, 1.0),
    ((9, 15, 27), 1e-9, 1, 3, 1.0), ((24, 25, 16), 1e-10, -1, 1, 1e200)])
def test_line_df_against_cufft(monkeypatch, ntype, modes, tol, iflag, ntr, scale):
    rng = np.random.default_rng(sum(modes) + ntype)
    M = 3000
    pts = NC.points(rng, len(modes), M, edges=False)
    data = (NC.strengths(rng, M, ntr) if ntype == 1 else NC.coeffs(rng, modes, ntr)) * scale
    kw = dict(ntr=ntr, iflag=iflag, maxbatchsize=2)
    monkeypatch.setenv("CUFINUFFT_FP64_DF_FFT", "0")
    ref, _ = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw)
    monkeypatch.delenv("CUFINUFFT_FP64_DF_FFT")
    out, info = NC.run_gpu(ntype, modes, pts, data, tol, False, **kw)
    assert np.linalg.norm(out / scale - ref / scale) / np.linalg.norm(ref / scale) < 1e-13, info
