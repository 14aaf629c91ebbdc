"""complex64 device arrays at an odd element of a larger array: their addresses
are multiples of 8 bytes only, which is all that the type asks for.  Every call
gives the same bits there as on arrays that torch allocated (multiples of 512)."""
import ctypes as C

import numpy as np
import pytest
import torch

import fame
from fame import _lib as L

pytestmark = pytest.mark.gpu


def shifted(nvec, length):
    """(nvec, length) complex64, one element into its allocation."""
    a = torch.zeros(1 + nvec * length, dtype=torch.complex64, device="cuda")[1:].view(nvec, length)
    assert a.data_ptr() % 16 == 8
    return a


def ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,nvec", [(4, 1), (6, 2), (10, 3), (24, 2)])
@pytest.mark.parametrize("precond", [True, False])
def test_solve_writes_any_array(cuda, fame_lib, n, nvec, precond):
    plan = fame.woodpile_plan(n, fame.band_path(npts=40)[1:2])
    plan.set_option("precond", precond)
    length = 4 * n ** 3
    b = torch.randn(nvec, length, dtype=torch.complex64, device="cuda")
    b2, y, y2 = shifted(nvec, length), torch.empty_like(b), shifted(nvec, length)
    b2.copy_(b)
    plan._stream()
    for src, dst in ((b, y), (b2, y2)):
        rc = fame_lib.fame_apply_Binv(plan.raw, L.FAME_C64, ptr(src), ptr(dst), nvec, None, 1e-4, 2000, None, None, 0)
        assert rc == L.FAME_OK
    assert torch.equal(y2, y)
    assert float(torch.linalg.norm(y)) > 0.0


@pytest.mark.parametrize("n", [4, 10, 24])
def test_operators_take_any_array(cuda, fame_lib, n):
    plan = fame.woodpile_plan(n, fame.band_path(npts=40)[1:2])
    nq, nvec = n ** 3, 3
    h = plan.raw
    calls = {
        "A": (4, 4, lambda x, y: fame_lib.fame_apply_A(h, L.FAME_C64, x, y, nvec, None, 0)),
        "B": (4, 4, lambda x, y: fame_lib.fame_apply_B(h, L.FAME_C64, x, y, nvec, None, 0)),
        "material": (6, 6, lambda x, y: fame_lib.fame_apply_material(h, L.FAME_C64, x, y, nvec, None, 0)),
    }
    for t in (0, 1):
        calls["transform", t] = (3, 3, lambda x, y, t=t: fame_lib.fame_curl_transform(h, L.FAME_C64, t, x, y, nvec,
                                                                                   None, 0))
    for w in range(4):
        calls["handle", w] = (2 if w < 2 else 3, 3 if w < 2 else 2,
                              lambda x, y, w=w: fame_lib.fame_apply_handle(h, L.FAME_C64, w, x, y, nvec, None, 0))
    plan._stream()
    for name, (ni, no, call) in calls.items():
        x = torch.randn(nvec, ni * nq, dtype=torch.complex64, device="cuda")
        y = torch.empty(nvec, no * nq, dtype=torch.complex64, device="cuda")
        x2, y2 = shifted(nvec, ni * nq), shifted(nvec, no * nq)
        x2.copy_(x)
        assert call(ptr(x), ptr(y)) == L.FAME_OK and call(ptr(x2), ptr(y2)) == L.FAME_OK, name
        assert torch.equal(y2, y), name
