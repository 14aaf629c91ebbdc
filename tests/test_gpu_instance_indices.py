"""Instance indices of a call travel in the kernel arguments up to 128 vectors and
in device memory beyond, or with more than 256 instances: a vector's result is
the same either way, for every call that takes them."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("nk", [3, 300])
def test_indices_in_arguments_and_memory(cuda, fame_lib, nk, dtype):
    n = 6
    rng = np.random.default_rng(nk)
    tens = np.zeros((nk, 2, 27), dtype=np.complex128)
    for k in range(nk):
        for p in range(2):
            tens[k, p, 0:9] = ((1.0 + 5.0 * p + 0.01 * k) * np.eye(3)).ravel()
            tens[k, p, 9:18] = np.eye(3).ravel()
            tens[k, p, 18:27] = (0.1j * p * np.eye(3)).ravel()
    plan = fame.Plan(n, rng.uniform(0.3, 2.5, size=(nk, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8), tens)
    nq, nvec = n ** 3, 140
    inst = rng.integers(0, nk, nvec).astype(np.int32)
    inst[:2] = 0, nk - 1
    x = torch.randn(nvec, 6 * nq, dtype=dtype, device="cuda")
    calls = [(plan.apply_A, 4), (plan.apply_B, 4), (plan.material, 6),
             (lambda v, i: plan.transform(v, 0, inst=i), 3), (lambda v, i: plan.transform(v, 1, inst=i), 3),
             (lambda v, i: plan.handle(1, v, inst=i), 2), (lambda v, i: plan.handle(3, v, inst=i), 3)]
    if dtype == torch.complex128:
        om = np.linspace(0.3, 1.2, nvec)
        calls.append((lambda v, i: torch.cat([plan.restore(v, om[:len(v)], inst=i)[q] for q in "EH"], dim=1), 4))
    for j, (f, m) in enumerate(calls):
        v = x[:, :m * nq].contiguous()
        one = torch.cat([f(v[k:k + 1], inst[k:k + 1]) for k in range(0, nvec)])
        for width in (33, 128, 129, 140):
            assert torch.equal(f(v[:width], inst[:width]).reshape(width, -1), one.reshape(nvec, -1)[:width]), (j, width)


def test_indices_outlive_the_callers_array(cuda, fame_lib):
    """The library may copy the indices after the call has returned: from memory of
    its own, with the caller's array overwritten or freed by then, however many
    calls are under way."""
    n, nk, nvec = 8, 3, 900
    rng = np.random.default_rng(5)
    plan = fame.Plan.from_phases(n, rng.uniform(0.3, 2.5, size=(nk, 3)), rng.integers(0, 2, n ** 3).astype(np.uint8),
                                 [fame.bi_isotropic(1.0, 0.0), fame.bi_isotropic(13.0, 0.4)])
    x = torch.randn(nvec, 4 * n ** 3, dtype=torch.complex64, device="cuda")
    whole = [plan.apply_A(x, inst=k) for k in range(nk)]
    outs = {}
    for j in range(200):  # 180000 indices: more than one turn of the library's buffer
        inst = ((np.arange(nvec) + j) % nk).astype(np.int32)
        y = plan.apply_A(x, inst=inst)
        if j % 20 == 0:
            outs[j] = y
        inst[:] = 0
    for j, y in outs.items():
        want = (np.arange(nvec) + j) % nk
        for k in range(nk):
            assert torch.equal(y[torch.from_numpy(want == k).cuda()], whole[k][torch.from_numpy(want == k).cuda()]), (j, k)
