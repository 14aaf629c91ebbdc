"""What fame_get_tune reports for a width with nothing installed is what runs,
so that installing it changes nothing."""
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


def launches(lib, f):
    before = lib.fame_kernel_launches()
    y = f()
    return lib.fame_kernel_launches() - before, y


@pytest.mark.parametrize("n,nvec,halves", [(24, 161, True), (60, 10, True), (30, 80, True), (24, 8, False), (24, 400, False)])
def test_reported_default_is_the_one_that_runs(cuda, fame_lib, n, nvec, halves):
    plan = fame.woodpile_plan(n, fame.band_path(npts=40)[1:2])
    x = torch.randn(nvec, 4 * n ** 3, dtype=torch.complex64, device="cuda")
    t = plan.get_tune("c64", nvec)
    assert t["chunk"] == ((nvec + 1) // 2 if halves else 0) and t["stencil_tpb"] == 0
    count, y = launches(fame_lib, lambda: plan.apply_B(x))
    assert count == (10 if halves else 5)
    plan.set_tune("c64", nvec, t["chunk"], t["stencil_tpb"], t["lanes"])
    again, y2 = launches(fame_lib, lambda: plan.apply_B(x))
    assert again == count and torch.equal(y2, y)
    plan.set_tune("c64", nvec, 0, 0)  # the whole batch
    whole, y3 = launches(fame_lib, lambda: plan.apply_B(x))
    assert whole == 5 and torch.equal(y3, y)
