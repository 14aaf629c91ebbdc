"""Solves of batches wide enough that a vector has a few CTAs of its own only."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


# The recurrence's residual is below tol at the end; the true one differs by the
# rounding of some dozen updates: 1e2 * 1e2 units, 1e-12 and 1e-3 against tol.
@pytest.mark.parametrize("dtype,tol", [(torch.complex128, 1e-8), (torch.complex64, 3e-3)])
@pytest.mark.parametrize("n,nvec", [(4, 160), (12, 40), (16, 77), (20, 153), (12, 305), (24, 20)])
@pytest.mark.parametrize("precond", [True, False])
def test_every_vector_is_solved(cuda, fame_lib, n, nvec, dtype, tol, precond):
    rng = np.random.default_rng(n)
    plan = fame.Plan.from_phases(n, rng.uniform(0.3, 2.5, size=(2, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8),
                                 [fame.bi_isotropic(1.0, 0.0), fame.bi_isotropic(13.0, 0.3)])
    plan.set_option("precond", precond)
    b = torch.randn(nvec, 4 * n ** 3, dtype=dtype, device="cuda")
    inst = rng.integers(0, 2, nvec).astype(np.int32)
    x, its, rr = plan.apply_Binv(b, tol=tol, maxit=3000, inst=inst)
    r = b.to(torch.complex128) - plan.apply_B(x.to(torch.complex128), inst)
    rel = torch.linalg.norm(r, dim=1) / torch.linalg.norm(b.to(torch.complex128), dim=1)
    assert float(rel.max()) < 2 * tol
    assert np.all((0 < its) & (its < 3000)) and np.all(rr <= tol)
