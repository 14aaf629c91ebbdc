"""FP64 and double-single operators without the plan's Pi table, where the three
field CTAs of a plane share its evaluation, against the same with the table."""
import ctypes as C

import numpy as np
import pytest
import torch

import fame
from fame import _lib as L

pytestmark = pytest.mark.gpu

SIZES = (4, 6, 8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 60, 64)


@pytest.mark.parametrize("n,prec", [(n, L.FAME_C128) for n in SIZES] + [(n, L.FAME_C128_DS) for n in (12, 24, 40, 48, 60)])
def test_evaluated_pi_equals_the_table(cuda, fame_lib, n, prec):
    """Both evaluate the same expressions, in FP64 or, evaluated in double-single, to
    2^-47; |L|^2 - |L.w|^2 loses up to some hundred units of either at a few voxels:
    1e-13 and 1e-12 of the norm."""
    rng = np.random.default_rng(n)
    nk, nvec = 2, 3
    plan = fame.Plan.from_phases(n, rng.uniform(0.3, 2.5, size=(nk, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8),
                                 [fame.bi_isotropic(1.0, 0.0), fame.bi_isotropic(13.0, 0.4)])
    x = torch.randn(nvec, 4 * n ** 3, dtype=torch.complex128, device="cuda")
    inst = np.array([1, 0, 1], dtype=np.int32)
    ys = []
    for table in (True, False):
        plan.set_option("pi_table", table)
        y = torch.empty_like(x)
        plan._stream()
        rc = fame_lib.fame_apply_B(plan.raw, prec, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), nvec,
                                   inst.ctypes.data, 0)
        assert rc == L.FAME_OK
        ys.append(y)
    err = torch.linalg.norm(ys[1] - ys[0], dim=1) / torch.linalg.norm(ys[0], dim=1)
    assert float(err.max()) < (1e-13 if prec == L.FAME_C128 else 1e-12)
