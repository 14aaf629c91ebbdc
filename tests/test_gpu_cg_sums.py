"""The norms of a complex64 solve do not depend on the width of its batch: the
FP32 part of a sum ends with a voxel, whatever the number of voxels that a
thread of a wide batch goes through."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [True, False])
@pytest.mark.parametrize("n,nvec", [(24, 250), (30, 200)])
def test_norm_of_a_constant_vector(cuda, fame_lib, n, nvec, precond):
    """Equal terms round the same way again and again once the sum is large (216
    of them: some 3e-6 of the sum).  One thread's 8 products of a voxel carry at
    most 8 units of 2^-24 of relative error, in a batch of one and of many, and
    the norm half of their sum's: 8 * 2^-24 for the difference of two."""
    rng = np.random.default_rng(n)
    plan = fame.Plan.from_phases(n, rng.uniform(0.3, 2.5, size=(1, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8),
                                 [fame.bi_isotropic(1.0, 0.0), fame.bi_isotropic(13.0, 0.4)])
    plan.set_option("precond", precond)
    worst = 0.0
    for t in (1.1, 1.2, 1.3):
        b = torch.full((1, 4 * n ** 3), t, dtype=torch.complex64, device="cuda")
        _, its, one = plan.apply_Binv(b, tol=1e-6, maxit=1)
        _, _, many = plan.apply_Binv(b.expand(nvec, -1), tol=1e-6, maxit=1, inst=np.zeros(nvec, np.int32))
        assert its[0] == 1 and 0.0 < one[0] < 10.0
        worst = max(worst, float(np.max(np.abs(many / one[0] - 1.0))))
    assert worst < 8 * 2.0 ** -24
