"""FP32 grids whose sides are powers of two transform by the pruned line passes
without being asked: against cuFFT with the mode-row kernel (CUFINUFFT_FFT=cufft:
any other name), every length from 256 to 4096 along either axis, even and odd mode
counts, both types and signs, batches with a partial last one."""
import numpy as np
import pytest

from tests import nufft_cases as NC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntype", [1, 2])
@pytest.mark.parametrize("iflag", [1, -1])
@pytest.mark.parametrize("modes", [(127, 2047), (2048, 128), (511, 512), (256, 1023), (1024, 255), (127, 128, 127)])
def test_against_cufft(monkeypatch, ntype, iflag, modes):
    import torch

    from cufinufft_gb300 import cufinufft
    rng = np.random.default_rng(sum(modes))
    M = 5000
    pts = [torch.from_numpy(p).cuda() for p in NC.points(rng, len(modes), M, dtype=np.float32, edges=False)]
    c = torch.from_numpy(np.stack([NC.strengths(rng, M, dtype=np.complex64) for _ in range(3)])).cuda()
    fk = torch.from_numpy(NC.coeffs(rng, modes, 3, dtype=np.complex64)).cuda()
    outs = []
    for form in (None, "cufft"):
        if form:
            monkeypatch.setenv("CUFINUFFT_FFT", form)
        plan = cufinufft(ntype, modes[::-1], n_trans=3, eps=1e-6, isign=iflag, dtype=np.float32, maxbatchsize=2)
        assert plan.info()["line_fft"] == (0 if form else 1)
        plan.set_pts(*pts[::-1])
        c2, f2 = c.clone(), fk.clone()
        plan.execute(c2, f2)
        torch.cuda.synchronize()
        outs.append((f2 if ntype == 1 else c2).cpu().numpy())
    # FP32 rounding of the FFT, amplified by the deconvolution at the mode corners
    assert np.linalg.norm(outs[0] - outs[1]) / np.linalg.norm(outs[1]) < 2e-6
