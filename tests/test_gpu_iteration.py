"""The kernels of the solver iterations where their forms change: the FP32
operator of every order with its tails, the direction update inside it, solves
stopped at every early iteration, the coarse solve on either side of its
shared-memory limit, the Jacobi diagonal, Dirichlet masks in the weights, and
the optimiser's constraint counts."""
import numpy as np
import pytest
import torch

import test_gpu_fixed_point as fixed
from oracle import schwarz_ref
from oracle.mma_ref import MMA

pytestmark = pytest.mark.gpu

EPS32 = 2.0 ** -24


def T(a, dev, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype)


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("E", [(1, 1, 1), (3, 1, 1), (9, 3, 1)])
def test_fp32_operator(pkg, orc, dev, lx, E):
    """Element counts off every block's size; both paths of lx = 8."""
    c = pkg.coef_t.box(*E, lx, amp=0.04, seed=3, device=dev)
    m = {k: t.cpu().numpy() for k, t in c.geometry().items()}
    m.update(lx=lx, E=E[0] * E[1] * E[2], n=c.n)
    c.set_coefs(h1c=0.5)
    u = np.random.default_rng(lx).standard_normal(c.n).astype(np.float32)
    ref, bound = fixed.contract(m, orc.gll(lx)[2].reshape(lx, lx), u.astype(np.float64), np.longdouble(0.5))
    for tma in (True, False):
        c.set_ax_path(tma)
        w = torch.full((c.n,), float("nan"), dtype=torch.float32, device=dev)
        pkg.ax_helm_t().compute(w, T(u, dev, torch.float32), c)
        torch.cuda.synchronize()
        # lx + 3 terms a sum, two sums, matrix, metric and product rounded to FP32: (2 lx + 12) roundings
        assert np.all(abs(w.cpu().numpy() - ref) <= (2 * lx + 12) * EPS32 * bound)


def reference_cg(pkg, c, sw, f, mult, mask, steps, dev):
    """x after each step of the preconditioned iteration, in FP64 torch around the library's FP64 operator."""
    def M(r):
        z = torch.empty(c.n, dtype=torch.float32, device=dev)
        sw.apply(z, r.float())
        return z.double()

    x, r = torch.zeros_like(f), f.clone()
    z = M(r)
    p, rz, w, out = z.clone(), (r * z * mult).sum(), torch.empty_like(f), []
    for _ in range(steps):
        pkg.ax_helm_t().compute(w, p, c)
        pkg.gs_t(c).op(w)
        pkg.api.bc_list_apply_scalar(c, w)
        alpha = rz / (p * w * mult).sum()
        x = x + alpha * p
        r = r - alpha * w
        z = M(r)
        new = (r * z * mult).sum()
        p, rz = z + (new / rz) * p, new
        out.append(x.clone())
    return out


@pytest.mark.parametrize("lx,tma", [(4, True), (6, True), (8, True), (8, False)])
@pytest.mark.parametrize("h1,h2", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("general", [False, True])
def test_stopped_solves(pkg, orc, dev, lx, tma, h1, h2, general):
    """A solve capped at k iterations returns the k-th iterate: every step's
    x += alpha p is there, whichever kernel does it."""
    E = (3, 2, 1)
    c = pkg.coef_t.box(*E, lx, amp=0.04, seed=4, device=dev)
    mask = orc.mask_face_xmax(*E, lx)
    c.set_mask(T(mask, dev, torch.int32), base=1)
    rng = np.random.default_rng(lx)
    kw = {}
    if h1:
        kw["h1"] = T(rng.uniform(0.5, 1.5, c.n), dev)
    if h2:
        kw.update(h2=T(rng.uniform(0.0, 5.0, c.n), dev), ifh2=True)
    c.set_coefs(**kw)
    c.set_ax_path(tma)
    ones = torch.ones(c.n, dtype=torch.float64, device=dev)
    pkg.gs_t(c).op(ones)
    f = c.rhs_assemble(T(rng.standard_normal(c.n), dev))
    sw = pkg.schwarz_t(c, coarse=not general, general=general)
    ref = reference_cg(pkg, c, sw, f, 1.0 / ones, mask, 4, dev)
    for k in range(1, 5):
        ksp = pkg.krylov_solver_factory(c, "cg_mixed", k, 1e-14)
        ksp.set_inner(1e-12, 1)  # no residual replacement on the way
        ksp.set_schwarz(sw)
        x = torch.zeros_like(f)
        mon = ksp.solve(x, f)
        torch.cuda.synchronize()
        assert mon.iter == k, mon
        # a step's FP32 roundings are some 1e2 * 2^-24 of its vectors; a missing step moves x by percents
        assert float((x - ref[k - 1]).norm()) <= 1e-4 * float(ref[k - 1].norm()), k


# inside and outside the shared memory of a plane (x, y) and of a column (z)
@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 0.0, False), (5, 7, 3, 4, 0.05, True), (216, 2, 2, 4, 0.0, True),
                                   (230, 2, 2, 4, 0.0, True), (2, 2, 148, 4, 0.0, True), (2, 2, 156, 4, 0.0, True)])
def test_coarse_solve_sizes(pkg, orc, dev, shape):
    ex, ey, ez, lx, amp, dirichlet = shape
    m = orc.build_mesh(ex, ey, ez, lx, amp=amp, seed=2)
    c = pkg.coef_t.box(ex, ey, ez, lx, amp=amp, seed=2, device=dev)
    mask = orc.mask_face_xmax(ex, ey, ez, lx) if dirichlet else None
    if dirichlet:
        c.set_mask(T(mask, dev, torch.int32), base=1)
    rng = np.random.default_rng(5)
    h2 = rng.uniform(0.0, 2.0, m.n)
    c.set_coefs(h1c=0.5, h2=T(h2, dev), ifh2=True)
    sw = pkg.schwarz_t(c, coarse=True)
    g = orc.gs_op(m, rng.standard_normal(m.n)) * m.mult
    r = (orc.apply_mask_zero(g, mask) if dirichlet else g).astype(np.float32)
    z = torch.empty(m.n, dtype=torch.float32, device=dev)
    sw.apply(z, T(r, dev, torch.float32))
    torch.cuda.synchronize()
    ref = schwarz_ref.apply(m, r.astype(np.float64), (ex, ey, ez), h1=0.5, h2=h2, mask=mask, coarse=True)
    # the local solves' 2e-5, and six FP32 transforms whose sums are as long as the grid
    tol = 2e-5 + 6 * max(ex, ey, ez) * EPS32
    assert np.linalg.norm(z.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("field", [False, True])
def test_jacobi_diagonal(pkg, orc, dev, lx, field):
    """Against extended precision on the library's own metrics."""
    E, Q = (3, 2, 1), np.longdouble
    m = orc.build_mesh(*E, lx, amp=0.05, seed=6)
    c = pkg.coef_t.box(*E, lx, amp=0.05, seed=6, device=dev)
    G = {k: t.cpu().numpy().astype(Q).reshape(6, lx, lx, lx) for k, t in c.geometry().items() if t.numel() == c.n}
    rng = np.random.default_rng(lx)
    h2 = rng.uniform(0.0, 2.0, m.n)
    h1 = rng.uniform(0.5, 1.5, m.n) if field else None
    c.set_coefs(h1=None if h1 is None else T(h1, dev), h1c=0.75, h2=T(h2, dev), ifh2=True)
    jac = pkg.api.jacobi_t(c)
    jac.update()
    h = np.full(m.n, 0.75) if h1 is None else h1
    h = h.astype(Q).reshape(6, lx, lx, lx)
    D = orc.gll(lx)[2].reshape(lx, lx).astype(Q)
    D2, d = D * D, np.diag(D)
    e = lambda v, ax: v.reshape([1] + [lx if q == ax else 1 for q in (1, 2, 3)])
    main = (np.einsum("li,ekjl->ekji", D2, h * G["g11"]) + np.einsum("lj,ekli->ekji", D2, h * G["g22"])
            + np.einsum("lk,elji->ekji", D2, h * G["g33"]))
    i, j, k = e(d, 3), e(d, 2), e(d, 1)
    cross = [2 * h * i * j * G["g12"], 2 * h * i * k * G["g13"], 2 * h * j * k * G["g23"]]
    mass = (m.B * h2).astype(Q).reshape(main.shape)
    ids = np.unique(m.gid, return_inverse=True)[1].ravel()

    def assembled(v):
        t = np.zeros(ids.max() + 1, dtype=Q)
        np.add.at(t, ids, v.ravel())
        return t[ids]

    diag, size = assembled(main + sum(cross) + mass), assembled(main + sum(map(abs, cross)) + mass)
    # D within 8 roundings an entry (squared: 16), the mass within 32, 3 lx + 4 terms, the products, the assembly
    got = jac.dinv().cpu().numpy().astype(Q)
    assert np.all(abs(got * diag - 1) <= (3 * lx + 64) * Q(2.0) ** -53 * size / diag)


def test_mask_entries_and_changes(pkg, orc, dev):
    """A mask with repeated entries, and one set after a solve under another,
    act as the mask by itself on a new mesh: the same iterates, bit for bit."""
    E, lx = (4, 3, 2), 5
    mask = orc.mask_face_xmax(*E, lx)
    f = T(np.random.default_rng(2).standard_normal(24 * lx ** 3), dev)

    def solve(c, m):
        c.set_mask(T(m, dev, torch.int32), base=1)
        c.set_coefs(h1c=1.0, h2c=0.5, ifh2=True)
        x = torch.zeros_like(f)
        mon = pkg.krylov_solver_factory(c, "cg", 40, 1e-11).solve(x, c.rhs_assemble(f))
        torch.cuda.synchronize()
        assert mon.iter == 40, mon
        assert not x[torch.from_numpy(m.astype(np.int64) - 1).to(dev)].any()
        return x

    new = lambda: pkg.coef_t.box(*E, lx, amp=0.05, seed=7, device=dev)
    c, ref = new(), solve(new(), mask)
    assert torch.equal(solve(c, np.concatenate([mask, mask[:7], mask[3:]])), ref)
    half = solve(c, mask[: mask.size // 2])
    assert torch.equal(half, solve(new(), mask[: mask.size // 2])) and not torch.equal(half, ref)
    assert torch.equal(solve(c, mask), ref)


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [5, 777])
def test_mma_constraint_counts(pkg, dev, m, n):
    rng = np.random.default_rng(10 * m + n)
    w, V = rng.uniform(0.5, 2.0, n), rng.uniform(0.1, 1.0, (m, n))
    lim = 0.4 * V.mean(axis=1)

    def prob(x):
        return -w / x ** 2 / n, (V * x).mean(axis=1) - lim, V / n

    x0 = np.full(n, 0.5)
    ref = MMA(x0, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0)
    xd, xr = T(x0, dev), x0.copy()
    opt = pkg.mma_t(xd, n, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0)
    for it in range(1, 5):
        df0, f, df = prob(xd.cpu().numpy())
        opt.update(it, xd, T(df0, dev), f, T(df.T.ravel(), dev))
        df0, f, df = prob(xr)
        xr = ref.update(it, xr, df0, f, df)
        # the same Newton steps; their rounding grows with the condition of the m x m system (some 1e4)
        assert np.allclose(xd.cpu().numpy(), xr, rtol=1e-8, atol=1e-10)
