"""Performance cases of the eigensolver: what a user has it do, over the real
range of grid sizes, batch widths, precisions and directions.

The crystals are woodpiles (FCC, rods of width 0.25 a, eps 13, chirality
gamma) at generic wave vectors, the fields of the adjoint cases a continuous
chiral medium.  Every case goes through the package's public entry points;
``exact`` restates the operators in plain complex128 torch.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "3d-bi-anisotropic-phc_gb300"))

import fame  # noqa: E402

DTYPE = {"c64": torch.complex64, "c128": torch.complex128}
BYTES = {"c64": 8, "c128": 16}
# grid sizes with a compiled transform, from the smallest a band path is run on
SIZES = (12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 60, 64)
LATTICE = 0.5 * np.array([[0.0, 1.0, 1.0], [1.0, 0.0, 1.0], [1.0, 1.0, 0.0]])  # FCC, columns


def listed():
    return [
        # One operator application on the CPU-sized grid (24^3, one k-point):
        # the smallest call, a step of a user's own Krylov loop.
        dict(name="fncB c64 n24 one", kind="fncB", prec="c64", n=24, nk=1, per=1),
        # The operator on the benchmark grid, ten k-points of a band path in
        # lock step: what a batched band solve spends its time on.
        dict(name="fncB c64 n60 ten", kind="fncB", prec="c64", n=60, nk=10, per=1),
        # A grid of 2 x 25 points per axis and an odd block of vectors of one
        # k-point, as a block residual check applies it.
        dict(name="fncB c64 n50 block", kind="fncB", prec="c64", n=50, nk=1, per=3),
        # The operator in double precision: the reference's own form and every
        # reported residual.
        dict(name="fncB c128 n40 four", kind="fncB", prec="c128", n=40, nk=4, per=1),
        # B^{-1} in single precision for eight k-points at once: the inner
        # solve of an interior search, or of a user's own Lanczos.
        dict(name="fncinvB c64 n48 eight", kind="fncinvB", prec="c64", n=48, nk=8, per=1),
        # B^{-1} in double precision at the reference's tolerance.
        dict(name="fncinvB c128 n30 two", kind="fncinvB", prec="c128", n=30, nk=2, per=1),
        # The curl transform there and back (MtxVecMul_FFT, both directions).
        dict(name="transform c128 n36 five", kind="transform", prec="c128", n=36, nk=5, per=1),
        # The composed handles with the material operator between them, the
        # way code written against the reference's closures calls them.
        dict(name="handles c64 n32 four", kind="handles", prec="c64", n=32, nk=2, per=2),
        # E and H fields, the residual and the field maxima of a k-point's
        # eight eigenvectors after a solve.
        dict(name="restore n40 eight", kind="restore", prec="c128", n=40, nk=1, per=8),
        # Backward pass of the eigenfrequencies: the gradient of three bands
        # at four k-points with respect to the per-vertex fields.
        dict(name="gradient n40 four", kind="gradient", prec="c128", n=40, nk=4, per=3),
        # A whole band solve in double precision on a small grid.
        dict(name="bands c128 n16 two", kind="bands", prec="c128", n=16, nk=2, bands=6),
        # A whole mixed-precision band solve of four k-points of the zone.
        dict(name="bands c64 n40 four", kind="bands", prec="c64", n=40, nk=4, bands=8),
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        c = _draw(rng)
        if c not in known:
            return c


def _draw(rng):
    kind = rng.choices(("fncB", "fncinvB", "transform", "handles", "restore", "gradient", "bands"),
                       weights=(6, 4, 2, 2, 1, 1, 2))[0]
    prec = "c128" if kind in ("restore", "gradient") else rng.choice(("c64", "c64", "c128"))
    if kind == "bands":
        n = rng.choice((12, 16, 18, 20, 24, 30) if prec == "c64" else (12, 16))
        return dict(kind=kind, prec=prec, n=n, nk=rng.randint(1, 4 if prec == "c64" else 2),
                    bands=rng.randint(4, 8 if prec == "c64" else 6))
    big = {"fncB": 10 * 60 ** 3, "fncinvB": 8 * 48 ** 3, "transform": 10 * 60 ** 3, "handles": 10 * 48 ** 3,
           "restore": 8 * 40 ** 3, "gradient": 12 * 40 ** 3}[kind]
    if prec == "c128" and kind in ("fncB", "fncinvB"):
        big //= 8  # the double-precision arithmetic costs about that much more
    n = rng.choice([s for s in SIZES if s ** 3 <= big])
    most = max(1, min(16, big // n ** 3))
    nvec = int(round(math.exp(rng.uniform(0.0, math.log(most + 0.49)))))
    if kind == "gradient":
        per = rng.randint(1, min(4, nvec))
        return dict(kind=kind, prec=prec, n=n, nk=max(1, nvec // per), per=per)
    nk = rng.choice([d for d in range(1, nvec + 1) if nvec % d == 0])
    return dict(kind=kind, prec=prec, n=n, nk=nk, per=nvec // nk)


# -- inputs -----------------------------------------------------------------
def _phase(n):
    """Woodpile rods (half-width in the diagonal coordinate sqrt(2)/2 * 0.25)."""
    c = np.arange(n) / n
    c3, c2, c1 = np.meshgrid(c, c, c, indexing="ij")
    pos = np.stack([c1.ravel(), c2.ravel(), c3.ravel()], axis=1) @ LATTICE.T
    z, t1, t2, h = pos[:, 2], pos[:, 1] - pos[:, 0], pos[:, 1] + pos[:, 0], math.sqrt(2.0) / 2.0 * 0.25

    def rod(t, *centres):
        return np.any([np.abs(t - m) <= h for m in centres], axis=0)

    layer = np.minimum((z * 4.0).astype(int), 3)
    inside = np.select([layer == 0, layer == 1, layer == 2, layer == 3],
                       [rod(t1, -1.0, 0.0, 1.0), rod(t2, 0.5, 1.5), rod(t1, -0.5, 0.5), rod(t2, 0.0, 1.0, 2.0)])
    return inside.astype(np.uint8)


def _thetas(rng, nk):
    """Bloch angles of generic wave vectors, away from Gamma."""
    return rng.uniform(0.25, 0.9, size=(nk, 3)) * np.pi * rng.choice([-1.0, 1.0], size=(nk, 3))


def _constitutive(eps, gamma):
    c = np.zeros((6, 6), dtype=np.complex128)
    c[range(3), range(3)] = eps
    c[range(3, 6), range(3, 6)] = 1.0
    c[range(3), range(3, 6)] = 1j * gamma
    c[range(3, 6), range(3)] = -1j * gamma
    return c


def _host(case, seed):
    """The host-side inputs of a case: Bloch angles, and the crystal."""
    rng = np.random.default_rng(seed)
    d = dict(n=case["n"], nk=case["nk"], thetas=_thetas(rng, case["nk"]))
    if case["kind"] == "gradient":
        n = case["n"]
        q = np.arange(n) * (2 * np.pi / n)
        s = np.zeros((n, n, n))
        for _ in range(6):  # a smooth random field
            k = rng.integers(-2, 3, size=3)
            s += rng.normal() * np.cos(k[0] * q[None, None, :] + k[1] * q[None, :, None] + k[2] * q[:, None, None]
                                       + rng.uniform(0, 2 * np.pi))
        s = 1.0 / (1.0 + np.exp(-2.0 * s.ravel()))
        d.update(eps=1.0 + 12.0 * s, gamma=0.2 * s)
    else:
        d.update(phase=_phase(case["n"]), gammas=rng.uniform(0.05, 0.5, size=case["nk"]))
    return d


def _vectors(case, seed, blocks):
    """Unit-scale complex Gaussian vectors of `blocks` n^3 grids each."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 12345)
    shape = (case["nk"] * case["per"], blocks * case["n"] ** 3)
    real = torch.float32 if case["prec"] == "c64" else torch.float64
    return torch.complex(*(torch.randn(shape, generator=g, device="cuda", dtype=real) for _ in range(2)))


def _omegas(case, seed):
    rng = np.random.default_rng(seed + 777)
    om = np.sort(rng.uniform(0.2, 1.5, size=(case["nk"], case["per"])), axis=1)
    return om, rng.uniform(-1.0, 1.0, size=om.shape)


def prepare(case, seed):
    h = _host(case, seed)
    if case["kind"] == "gradient":
        plan = fame.Plan.from_fields(h["n"], h["thetas"], h["eps"], h["gamma"], LATTICE)
    else:
        air = _constitutive(1.0, 0.0)
        plan = fame.Plan.from_phases(h["n"], h["thetas"], h["phase"],
                                     [[air, _constitutive(13.0, g)] for g in h["gammas"]], LATTICE)
    s = dict(case=case, plan=plan)
    if case["kind"] == "bands":
        return s
    # vector v belongs to k-point v // per; None is the library's own order
    s["inst"] = None if case["per"] == 1 else np.repeat(np.arange(case["nk"], dtype=np.int32), case["per"])
    s["x"] = _vectors(case, seed, {"transform": 3}.get(case["kind"], 4))
    if case["kind"] in ("restore", "gradient"):
        s["x"] /= torch.linalg.vector_norm(s["x"], dim=1, keepdim=True)
        s["omega"], s["weight"] = _omegas(case, seed)
    if case["kind"] == "gradient":
        s["evs"] = list(s["x"].reshape(case["nk"], case["per"], -1))
    return s


# -- one pass ---------------------------------------------------------------
def run(s):
    case, plan = s["case"], s["plan"]
    kind = case["kind"]
    if kind == "bands":
        k = case["bands"]
        r = plan.band_solve(k, tol=1e-10, p=max(2 * k, 20), prec=case["prec"], inner_tol=1e-12)
        return r["omega"]
    x, inst = s["x"], s["inst"]
    if kind == "fncB":
        return fame.fncB(x, plan, inst)
    if kind == "fncinvB":
        return fame.fncinvB(x, plan, tol=1e-6 if case["prec"] == "c64" else 1e-12, inst=inst)
    if kind == "transform":
        return [fame.MtxVecMul_FFT(x, plan, "notranspose", inst), fame.MtxVecMul_FFT(x, plan, "transpose", inst)]
    if kind == "handles":
        half = 2 * plan.Nq
        u = plan.handle(0, x[:, :half], inst)
        v = plan.handle(1, x[:, half:], inst)
        w = plan.material(torch.cat([u, v], dim=1), inst)
        return [u, v, w, plan.handle(2, w[:, :3 * plan.Nq], inst), plan.handle(3, w[:, 3 * plan.Nq:], inst)]
    if kind == "restore":
        return plan.restore(x, s["omega"].reshape(-1), inst=inst)
    return list(fame.adjoint.gradient(plan, s["evs"], s["omega"], s["weight"]))


# -- what one pass cannot do without ------------------------------------------
def work(case):
    n, b = case["n"], BYTES[case["prec"]]
    nq = n ** 3
    fft = 15 * nq * math.log2(n)  # one 3-D transform of one field
    fncb = 12 * fft + 600 * nq    # six fields there and back, material tensors, Pi blocks
    if case["kind"] == "bands":
        steps = 4 * case["bands"] * case["nk"]  # Lanczos vectors, each one solve with B of some 30 products
        return {"bytes": steps * 8 * nq * 16, "flops": steps * 30 * fncb}
    nvec = case["nk"] * case["per"]
    if case["kind"] == "fncB":
        return {"bytes": nvec * 8 * nq * b, "flops": nvec * fncb}
    if case["kind"] == "fncinvB":
        return {"bytes": nvec * 8 * nq * b, "flops": nvec * fncb * (12 if case["prec"] == "c64" else 25)}
    if case["kind"] == "transform":
        return {"bytes": nvec * 9 * nq * b, "flops": nvec * 6 * fft}
    if case["kind"] == "handles":
        return {"bytes": nvec * 20 * nq * b, "flops": nvec * fncb}
    if case["kind"] == "restore":
        return {"bytes": nvec * 10 * nq * b, "flops": nvec * (6 * fft + 1000 * nq)}
    return {"bytes": nvec * 4 * nq * b + 32 * nq, "flops": nvec * (6 * fft + 400 * nq)}


# -- the same in plain complex128 torch -----------------------------------------
class _Ref:
    """The operators of one k-point: grids are [z, y, x], axis d of a shift -1 - d."""

    def __init__(self, n, theta, tensors):
        self.n, self.t = n, tensors  # t(block) -> [3][3] tensors per vertex, or scalars; blocks N, M, J
        j = torch.arange(n, device="cuda", dtype=torch.float64)
        th = [float(t) for t in theta]
        lam, self.S, self.tau = [], 1.0, []
        for d in range(3):
            view = [1, 1, 1]
            view[2 - d] = n
            a = (2 * math.pi * j + th[d]) / n
            lam.append(((torch.polar(torch.ones_like(a), a) - 1.0) * n).reshape(view).expand(n, n, n))
            self.S = self.S * torch.polar(torch.ones_like(j), j * th[d] / n).reshape(view)
            self.tau.append(complex(math.cos(th[d] / n), math.sin(th[d] / n)))
        L = torch.stack(lam)
        w = [c / math.sqrt(14.0) for c in (1.0, 2.0, 3.0)]
        p1 = torch.stack([w[2] * L[1].conj() - w[1] * L[2].conj(), w[0] * L[2].conj() - w[2] * L[0].conj(),
                          w[1] * L[0].conj() - w[0] * L[1].conj()])
        self.p1 = p1 / torch.sqrt((p1.abs() ** 2).sum(0))
        c, b = self.p1.conj(), L.conj()
        p2 = torch.stack([c[1] * b[2] - c[2] * b[1], c[2] * b[0] - c[0] * b[2], c[0] * b[1] - c[1] * b[0]])
        self.p2 = p2 / torch.sqrt((L.abs() ** 2).sum(0))

    def fields(self, x, bloch=False, side=None):
        """Spatial fields of [a1 b1 a2 b2] (or of one side's [a b])."""
        n, x = self.n, x.reshape(-1, self.n, self.n, self.n)
        out = []
        for s in (0, 1) if side is None else (side,):
            a, b = x[0], x[1]
            x = x[2:]
            f = b * self.p1.conj() - a * self.p2.conj() if s == 0 else a * self.p1 + b * self.p2
            out.append(torch.fft.ifftn(f, dim=(1, 2, 3)) * n ** 1.5)
        f = torch.cat(out)
        return f * self.S if bloch else f

    def coefs(self, f, bloch=False, side=None):
        f = torch.fft.fftn(f * self.S.conj() if bloch else f, dim=(1, 2, 3)) / self.n ** 1.5
        out = []
        for s in (0, 1) if side is None else (side,):
            g, f = f[:3], f[3:]
            out += [-(self.p2 * g).sum(0), (self.p1 * g).sum(0)] if s == 0 else \
                [(self.p1.conj() * g).sum(0), (self.p2.conj() * g).sum(0)]
        return torch.stack(out).reshape(-1)

    def up(self, g, d):    # (I + T_d) g
        return g + self.tau[d] * torch.roll(g, -1, dims=2 - d)

    def down(self, g, d):  # (I + T_d)^H g
        return g + self.tau[d].conjugate() * torch.roll(g, 1, dims=2 - d)

    def mean(self, a, *axes):
        for d in axes:
            a = 0.5 * (a + torch.roll(a, -1, dims=2 - d)) if isinstance(a, torch.Tensor) else a
        return a

    def material(self, f):
        """[M J^H; J N] on periodic-frame fields [u; v]."""
        N, M, J = (self.t(b) for b in range(3))
        oth = [(1, 2), (0, 2), (0, 1)]
        U = [0.25 * self.down(self.down(f[j], oth[j][0]), oth[j][1]) for j in range(3)]
        V = [0.5 * self.down(f[3 + j], j) for j in range(3)]
        out = []
        for i in range(3):
            h = sum(M[i][j] * U[j] for j in range(3) if j != i) + sum(J[j][i].conj() * V[j] for j in range(3))
            a, b = oth[i]
            out.append(self.mean(M[i][i].real, a, b) * f[i] + 0.25 * self.up(self.up(h, a), b))
        for i in range(3):
            h = sum(N[i][j] * V[j] for j in range(3) if j != i) + sum(J[i][j] * U[j] for j in range(3))
            out.append(self.mean(N[i][i].real, i) * f[3 + i] + 0.5 * self.up(h, i))
        return torch.stack(out)

    def B(self, x):
        return self.coefs(self.material(self.fields(x)))


def _refs(case, seed):
    h = _host(case, seed)
    n = case["n"]
    refs = []
    for k in range(case["nk"]):
        if case["kind"] == "gradient":
            tens = None
        else:
            ids = torch.from_numpy(h["phase"].astype(np.int64)).cuda().reshape(n, n, n)
            per = []
            for c in (_constitutive(1.0, 0.0), _constitutive(13.0, h["gammas"][k])):
                inv = np.linalg.inv(c)
                per.append([LATTICE.T @ q @ LATTICE for q in (inv[:3, :3], inv[3:, 3:], inv[:3, 3:])])
            blocks = [[[torch.tensor([per[0][b][i, j], per[1][b][i, j]], device="cuda")[ids] for j in range(3)]
                       for i in range(3)] for b in range(3)]
            tens = blocks.__getitem__
        refs.append(_Ref(n, h["thetas"][k], tens))
    return h, refs


def _cg(op, b):
    x, r = torch.zeros_like(b), b.clone()
    p, rho = r.clone(), torch.vdot(r, r).real
    goal = 1e-28 * rho
    for it in range(1, 2000):
        q = op(p)
        a = rho / torch.vdot(p, q).real
        x, r = x + a * p, r - a * q
        new = torch.vdot(r, r).real
        if it % 10 == 0 and new <= goal:
            break
        p, rho = r + (new / rho) * p, new
    return x


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "bands":
        return None  # a whole solve: no closed form, and a dense one takes too long
    h, refs = _refs(case, seed)
    x = _vectors(case, seed, {"transform": 3}.get(kind, 4)).to(torch.complex128)
    ref = [refs[v // case["per"]] for v in range(x.shape[0])]
    if kind == "fncB":
        return torch.stack([r.B(v) for r, v in zip(ref, x)])
    if kind == "fncinvB":
        return torch.stack([_cg(r.B, v) for r, v in zip(ref, x)])
    g = x.reshape(x.shape[0], -1, n, n, n)
    if kind == "transform":
        inv = [r.S * torch.fft.ifftn(f, dim=(1, 2, 3)) * n ** 1.5 for r, f in zip(ref, g)]
        fwd = [torch.fft.fftn(r.S.conj() * f, dim=(1, 2, 3)) / n ** 1.5 for r, f in zip(ref, g)]
        return [torch.stack([f.reshape(-1) for f in v]) for v in (inv, fwd)]
    if kind == "handles":
        f = [r.fields(v, bloch=True) for r, v in zip(ref, x)]
        w = [r.material(q * r.S.conj()) * r.S for r, q in zip(ref, f)]
        c = [r.coefs(q, bloch=True) for r, q in zip(ref, w)]
        f, w, c = (torch.stack([q.reshape(-1) for q in v]) for v in (f, w, c))
        m = 3 * n ** 3
        return [f[:, :m], f[:, m:], w, c[:, :2 * n ** 3], c[:, 2 * n ** 3:]]
    if kind in ("restore", "gradient"):
        x = _vectors(case, seed, 4)
        x /= torch.linalg.vector_norm(x, dim=1, keepdim=True)
        om, wt = (torch.from_numpy(a.reshape(-1)).cuda() for a in _omegas(case, seed))
    if kind == "restore":
        out = dict(E=[], H=[], res_orgsep=[], max_e=[], max_h=[])
        for r, v, o in zip(ref, x, om):
            def diff(f, d, r=r):   # n (T_d - I) f
                return n * (r.up(f, d) - 2.0 * f)

            def diff_h(f, d, r=r):
                return n * (r.down(f, d) - 2.0 * f)

            uv = r.material(r.fields(v))
            e, hh = -1j * uv[3:], -1j * uv[:3]
            curl = torch.stack([diff(e[2], 1) - diff(e[1], 2), diff(e[0], 2) - diff(e[2], 0),
                                diff(e[1], 0) - diff(e[0], 1)])
            curl_h = torch.stack([diff_h(hh[1], 2) - diff_h(hh[2], 1), diff_h(hh[2], 0) - diff_h(hh[0], 2),
                                  diff_h(hh[0], 1) - diff_h(hh[1], 0)])
            y = r.material(torch.cat([-curl, curl_h]))
            rs = torch.cat([y[3:] - 1j * o * e, y[:3] - 1j * o * hh])
            for key, val in zip(out, ((r.S * e).reshape(-1), (r.S * hh).reshape(-1),
                                      torch.linalg.vector_norm(rs), e.abs().max(), hh.abs().max())):
                out[key].append(val)
        return {key: torch.stack(val) for key, val in out.items()}
    eps, gam = (torch.from_numpy(h[q]).cuda().requires_grad_() for q in ("eps", "gamma"))
    G = LATTICE.T @ LATTICE
    total = 0.0
    for r, v, o, w in zip(ref, x, om, wt):
        a = 1.0 / (eps - gam ** 2)
        sc = [f.reshape(n, n, n) for f in (a, eps * a, -1j * gam * a)]
        r.t = lambda b, sc=sc: [[G[i, j] * sc[b].to(torch.complex128) for j in range(3)] for i in range(3)]
        f = r.fields(v)
        q = torch.vdot(f.reshape(-1), r.material(f).reshape(-1)).real
        total = total + w * o / q.detach() * q
    return list(torch.autograd.grad(total, (eps, gam)))
