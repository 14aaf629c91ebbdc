"""The material stencil's variants against each other: the product for real
N, M and imaginary J (bi-isotropic media) against the general complex one, at
the edges of the tiles (every row count of a CTA, ragged z-chunks, more phases
than the shared table holds), in both forms and both frames."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu

# two evaluations of the same sums in different orders: some 60 products and
# additions per output and a few hundred per DFT, each within one unit of rounding
TOL = {torch.complex64: 5e-6, torch.complex128: 1e-14}


def chiral_tensors(rng, nk, nphase):
    t = np.zeros((nk, nphase, 27), dtype=np.complex128)
    for k in range(nk):
        for p in range(nphase):
            for b in range(2):
                m = rng.standard_normal((3, 3))
                t[k, p, 9 * b:9 * b + 9] = (0.1 * (m + m.T) + (1.0 + p) * np.eye(3)).ravel()
            t[k, p, 18:] = 0.1j * rng.standard_normal(9)
    return t


@pytest.mark.parametrize("n,nphase", [(4, 1), (6, 2), (10, 3), (18, 2), (24, 9), (30, 2), (50, 2), (64, 2)])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_chiral_product_equals_the_general_one(cuda, fame_lib, n, nphase, dtype):
    rng = np.random.default_rng(n)
    nk = 2
    th = rng.uniform(-np.pi, np.pi, size=(nk, 3))
    phase = rng.integers(0, nphase, size=n ** 3).astype(np.uint8)
    chi = chiral_tensors(rng, nk, nphase)
    gen = chi.copy()
    gen[0, 0, 18] += 1e-150  # not imaginary: the general product, the same values
    plans = [fame.Plan(n, th, phase, t) for t in (chi, gen)]
    prec = "c64" if dtype == torch.complex64 else "c128"
    for nvec in (1, 3):
        x = torch.randn(nvec, 4 * n ** 3, dtype=dtype, device="cuda")
        w = torch.randn(nvec, 6 * n ** 3, dtype=dtype, device="cuda")
        for tpb in (0, 128):
            for p in plans:
                p.set_tune(prec, nvec, 0, tpb)
            a, b = (p.apply_B(x) for p in plans)
            assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < TOL[dtype], (nvec, tpb)
        a, b = (p.material(w) for p in plans)
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < TOL[dtype], nvec


@pytest.mark.parametrize("n", [10, 20, 36, 48])
def test_chunks_of_planes_do_not_change_a_result(cuda, fame_lib, n):
    """The single-pass stencil cuts z into chunks by the batch's width: every
    width gives a vector the same result to the last bit."""
    rng = np.random.default_rng(n)
    plan = fame.woodpile_plan(n, fame.band_path(npts=40)[1:2])
    plan.set_option("plane_split", False)
    x = torch.as_tensor(rng.standard_normal((21, 4 * n ** 3)) + 1j * rng.standard_normal((21, 4 * n ** 3)))
    x = x.to(torch.complex64).cuda()
    ref = plan.apply_B(x)
    for nvec in (1, 2, 5, 13):
        assert torch.equal(plan.apply_B(x[:nvec]), ref[:nvec]), nvec
