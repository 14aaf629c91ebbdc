"""The forms of a batched call that depend on its size: CG solves in both
precisions with and without the preconditioner, vectors that stop at different
iterations, batches with more instance indices than a kernel's arguments hold,
and gradients evaluated in several groups."""
import numpy as np
import pytest
import torch

import fame

pytestmark = pytest.mark.gpu


def plan_of(n, nk, seed=0):
    rng = np.random.default_rng(seed)
    th = rng.uniform(0.3, 2.5, size=(nk, 3))
    tens = np.zeros((nk, 2, 27), dtype=np.complex128)
    for p, eps in enumerate((1.0, 13.0)):
        tens[:, p, 0:9] = (eps * np.eye(3)).ravel()
        tens[:, p, 9:18] = np.eye(3).ravel()
        tens[:, p, 18:27] = (0.1j * p * np.eye(3)).ravel()
    return fame.Plan(n, th, rng.integers(0, 2, size=n ** 3).astype(np.uint8), tens)


# The recurrence's residual is below tol at the end; the true one differs by
# the rounding of some hundred updates of a solution some hundred times the
# right-hand side: 1e2 * 1e2 * eps, 1e-12 and 1e-3 against tol 1e-9 and 3e-3.
@pytest.mark.parametrize("dtype,tol", [(torch.complex128, 1e-9), (torch.complex64, 3e-3)])
@pytest.mark.parametrize("n,nvec", [(4, 1), (12, 5), (16, 2), (30, 3), (64, 1)])
@pytest.mark.parametrize("precond", [True, False])
def test_solve_leaves_its_residual(cuda, fame_lib, n, nvec, dtype, tol, precond):
    plan = plan_of(n, 1, seed=n)
    plan.set_option("precond", precond)
    g = torch.Generator().manual_seed(n)
    b = torch.randn(nvec, 4 * n ** 3, dtype=torch.complex128, generator=g)
    inst = np.zeros(nvec, dtype=np.int32)
    if nvec > 2:
        b[1] = 0  # never active
        e = torch.zeros(1, 4 * n ** 3, dtype=torch.complex128)
        e[0, 3] = 1e3
        b[2] = plan.apply_B(e.cuda(), inst[:1]).cpu()[0]  # stops at another iteration
    b = b.to(dtype).cuda()
    x, its, rr = plan.apply_Binv(b, tol=tol, maxit=5000, inst=inst)
    r = b.to(torch.complex128) - plan.apply_B(x.to(torch.complex128), inst)
    for v in range(nvec):
        if nvec > 2 and v == 1:
            assert not torch.any(x[v] != 0)
        else:
            assert float(torch.linalg.norm(r[v]) / torch.linalg.norm(b[v])) < 2 * tol, v
            assert 0 < its[v] < 5000 and rr[v] <= tol


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
@pytest.mark.parametrize("n", [8, 12])
def test_more_instances_than_the_arguments_hold(cuda, fame_lib, n, dtype):
    """33 and 40 vectors read their indices from memory, up to 32 from the
    kernel arguments: a vector's result is the same to the last bit."""
    plan = plan_of(n, 3, seed=1)
    x = torch.randn(40, 4 * n ** 3, dtype=dtype, device="cuda")
    inst = (np.arange(40) * 7 % 3).astype(np.int32)
    parts = torch.cat([plan.apply_B(x[a:a + 10], inst[a:a + 10]) for a in range(0, 40, 10)])
    for m in (32, 33, 40):
        assert torch.equal(plan.apply_B(x[:m], inst[:m]), parts[:m])


def test_gradient_in_groups(cuda, fame_lib):
    """Three k-points of 14 vectors make two groups; one call per k-point gives
    the same sums but for their order: 42 terms, some 1e-14 relative."""
    n, nk, per = 6, 3, 14
    rng = np.random.default_rng(4)
    plan = fame.Plan.from_fields(n, rng.uniform(0.3, 2.5, size=(nk, 3)), 1.0 + 12.0 * rng.random(n ** 3),
                                 0.2 * rng.random(n ** 3))
    ev = torch.randn(nk, per, 4 * n ** 3, dtype=torch.complex128, device="cuda")
    om, w = 0.2 + rng.random((nk, per)), rng.uniform(-1, 1, size=(nk, per))
    one = [torch.zeros(plan.Nq, dtype=torch.float64, device="cuda") for _ in range(2)]
    for k in range(nk):
        plan.eig_gradient(ev[k], om[k], w[k], inst=k, out=tuple(one), accumulate=True)
    for a, b in zip(fame.adjoint.gradient(plan, list(ev), om, w), one):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < 1e-12
    with pytest.raises(TypeError):
        fame.adjoint.gradient(plan, [ev[0], ev[1].to(torch.complex64), ev[2]], om, w)


@pytest.mark.parametrize("n", [4, 6, 24])
def test_preconditioner_inverts_a_homogeneous_medium(cuda, fame_lib, n):
    """One general Hermitian medium everywhere: fncB is then the 4x4 blocks that
    the preconditioner inverts, and the first iteration solves the system but
    for rounding (some hundred units of it, 1e-13; the bound is 1e-11)."""
    rng = np.random.default_rng(2)
    t = np.zeros((2, 1, 27), dtype=np.complex128)
    for k in range(2):
        for b in range(2):
            m = rng.standard_normal((3, 3)) + 1j * rng.standard_normal((3, 3))
            t[k, 0, 9 * b:9 * b + 9] = (0.1 * (m + m.conj().T) + (2.0 + b) * np.eye(3)).ravel()
        t[k, 0, 18:] = 0.1 * (rng.standard_normal(9) + 1j * rng.standard_normal(9))
    plan = fame.Plan(n, rng.uniform(0.3, 2.5, size=(2, 3)), np.zeros(n ** 3, np.uint8), t)
    b = torch.randn(2, 4 * n ** 3, dtype=torch.complex128, device="cuda")
    _, its, rr = plan.apply_Binv(b, tol=1e-11, maxit=50)
    assert np.all(np.asarray(its) == 1) and np.all(np.asarray(rr) < 1e-11)


@pytest.mark.parametrize("n,nvec", [(24, 161), (60, 10)])
def test_halves_of_a_large_batch(cuda, fame_lib, n, nvec):
    """A complex64 batch far beyond the L2 runs as two halves unless something is
    installed for its width: the same result to the last bit."""
    plan = plan_of(n, 1, seed=3)
    x = torch.randn(nvec, 4 * n ** 3, dtype=torch.complex64, device="cuda")
    inst = np.zeros(nvec, dtype=np.int32)
    y = plan.apply_B(x, inst)
    plan.set_tune("c64", nvec, 0, 0)
    assert torch.equal(plan.apply_B(x, inst), y)
