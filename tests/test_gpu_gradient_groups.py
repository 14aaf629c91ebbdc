"""fame.adjoint.gradient joins k-points for one call only while the joined copy
(and with it the plan's work arrays, three times as large) stays small."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk,per", [(6, 5, 3), (60, 2, 6), (60, 3, 6), (64, 4, 5), (64, 2, 16)])
def test_joined_copies_stay_small(cuda, fame_lib, n, nk, per):
    rng = np.random.default_rng(n)
    plan = fame.Plan.from_fields(n, rng.uniform(0.3, 2.5, size=(nk, 3)), 1.0 + 12.0 * rng.random(n ** 3),
                                 0.2 * rng.random(n ** 3))
    ev = torch.randn(nk, per, 4 * n ** 3, dtype=torch.complex128, device="cuda")
    om, w = 0.2 + rng.random((nk, per)), rng.uniform(-1, 1, size=(nk, per))
    calls = []
    eig_gradient = plan.eig_gradient

    def recorded(e, *a, **kw):
        calls.append((e.shape[0], e.numel() * 16, sorted(set(np.atleast_1d(kw["inst"]).tolist()))))
        return eig_gradient(e, *a, **kw)

    plan.eig_gradient = recorded
    g = fame.adjoint.gradient(plan, list(ev), om, w)
    assert sum(c[0] for c in calls) == nk * per
    for vectors, size, points in calls:
        assert len(points) == 1 or (size <= 192 << 20 and vectors <= 32)
    if 64 * plan.Nq * nk * per <= 192 << 20:
        assert len(calls) == 1  # small enough: all joined
    one = [torch.zeros(plan.Nq, dtype=torch.float64, device="cuda") for _ in range(2)]
    for k in range(nk):
        eig_gradient(ev[k], om[k], w[k], inst=k, out=tuple(one), accumulate=True)
    for a, b in zip(g, one):  # the same sums in another order: 32 terms, some 1e-14
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < 1e-12
