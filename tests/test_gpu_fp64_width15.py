"""FP64 type 1 at the widest kernels, whose own error comes near double-float rounding: no
further from the direct sums than with FP64 instructions (CUFINUFFT_FP64_DF=0).  Up to
width 14 the kernel's error, 3e-13 and more, covers the 5e-14 of the sums, the square of
whose ratio is under 0.03; the bound allows that and, near 1e-14, what the order of sums moves
(3e-16 between two runs of FP64 instructions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol,rule", [(1e-13, "tol"), (1e-13, "reference"), (1e-12, "tol")])
@pytest.mark.parametrize("modes,M", [((1001,), 20000), ((81, 60), 20000), ((18, 25, 20), 20000)])
def test_error_against_direct_sums(monkeypatch, modes, M, tol, rule):
    import torch

    from cufinufft_gb300 import cufinufft
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    pts = [(0.3 + 0.1 * torch.randn(M, generator=g, device="cuda", dtype=torch.float64)).clamp(-3, 3) for _ in modes]
    c = torch.randn(M, generator=g, device="cuda", dtype=torch.complex128)
    ref = torch.zeros(modes, dtype=torch.complex128, device="cuda")
    for s in range(0, M, 2000):
        e = [torch.exp(1j * torch.outer(p[s:s + 2000], torch.arange(n, device="cuda") - n // 2)) for p, n in zip(pts, modes)]
        t = c[s:s + 2000, None] * e[0]
        for f in e[1:-1]:
            t = (t[:, :, None] * f[:, None, :]).reshape(len(t), -1)
        ref += t.sum(0) if len(modes) == 1 else (t.T @ e[-1]).reshape(modes)
    err = []
    for df in (None, "0"):
        if df:
            monkeypatch.setenv("CUFINUFFT_FP64_DF", df)
        plan = cufinufft(1, modes, eps=tol, dtype=np.float64, width_rule=rule)
        plan.set_pts(*pts)
        fk = torch.zeros(modes, dtype=torch.complex128, device="cuda")
        plan.execute(c, fk)
        torch.cuda.synchronize()
        err.append(float((fk - ref).norm() / ref.norm()))
    print(modes, tol, rule, "error %.4e, FP64 instructions %.4e" % tuple(err))
    assert err[0] <= 1.03 * err[1] + 1e-15
