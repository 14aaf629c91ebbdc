"""The curl transform at every compiled grid size against torch's FFT (each
size has its own split of the pencils: prime-factor, Cooley-Tukey or none),
the handles as its composition with Pi, and complex64 against complex128."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu

SIZES = (4, 6, 8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 60, 64)
TOL = {torch.complex64: 2e-6, torch.complex128: 3e-15 * 4}  # a few rounding units per pass of log2(n^3) passes


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_transform_equals_fft(cuda, fame_lib, n, dtype):
    rng = np.random.default_rng(n)
    th = rng.uniform(-np.pi, np.pi, size=(2, 3))
    plan = fame.Plan(n, th, np.zeros(n ** 3, np.uint8), np.eye(3)[None].repeat(3, 0).reshape(1, 27))
    x = torch.randn(3, 3 * n ** 3, dtype=dtype, device="cuda")
    inst = np.array([0, 1, 1])
    j = torch.arange(n, device="cuda", dtype=torch.float64) / n
    for v in range(3):
        t = th[inst[v]]
        ph = [torch.polar(torch.ones_like(j), j * float(t[d])) for d in range(3)]
        S = ph[2][:, None, None] * ph[1][None, :, None] * ph[0][None, None, :]
        g = x[v].to(torch.complex128).reshape(3, n, n, n)
        for trans in (0, 1):
            ref = S * torch.fft.ifftn(g, dim=(1, 2, 3)) * n ** 1.5 if trans == 0 else \
                torch.fft.fftn(S.conj() * g, dim=(1, 2, 3)) / n ** 1.5
            got = plan.transform(x, trans, inst=inst)[v].to(torch.complex128).reshape(3, n, n, n)
            assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < TOL[dtype], (v, trans)


@pytest.mark.parametrize("n", SIZES)
def test_handles_and_fncB_across_precisions(cuda, fame_lib, n):
    rng = np.random.default_rng(n)
    plan = fame.Plan.from_phases(n, rng.uniform(0.3, 2.5, size=(2, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8),
                                 [fame.bi_isotropic(1.0, 0.0), fame.bi_isotropic(13.0, 0.4)])
    x = torch.randn(2, 4 * n ** 3, dtype=torch.complex128, device="cuda")
    x32 = x.to(torch.complex64)
    half = 2 * n ** 3
    eye = plan.handle(2, plan.handle(0, x[:, :half]))  # Prs Pr = I
    assert float(torch.linalg.norm(eye - x[:, :half]) / torch.linalg.norm(x[:, :half])) < 1e-13
    eye = plan.handle(3, plan.handle(1, x[:, half:]))
    assert float(torch.linalg.norm(eye - x[:, half:]) / torch.linalg.norm(x[:, half:])) < 1e-13
    for f in (plan.apply_B, lambda v: plan.handle(1, v[:, half:])):
        a, b = f(x32).to(torch.complex128), f(x)
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < 5e-6
    # the composition is the operator: B x = [Prs; Qrs] material [Pr; Qr] x
    w = plan.material(torch.cat([plan.handle(0, x[:, :half]), plan.handle(1, x[:, half:])], dim=1))
    m = 3 * n ** 3
    y = torch.cat([plan.handle(2, w[:, :m]), plan.handle(3, w[:, m:])], dim=1)
    b = plan.apply_B(x)
    assert float(torch.linalg.norm(y - b) / torch.linalg.norm(b)) < 1e-13
