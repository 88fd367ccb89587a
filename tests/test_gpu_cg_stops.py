"""FP64 and Schwarz-preconditioned CG stopped early: the last x += alpha p is
done, whichever kernel does it, on small meshes (dependent launches), just
below and above the size where those end, and where a block of the operator
takes several groups of elements."""
import numpy as np
import pytest
import torch

from test_gpu_iteration import T, reference_cg

pytestmark = pytest.mark.gpu


def plan(pkg, orc, dev, E, lx, h2c=3.0):
    c = pkg.coef_t.box(*E, lx, amp=0.04, seed=4, device=dev)
    c.set_mask(pkg.api.mask_face_xmax(*E, lx), base=1)
    c.set_coefs(h1c=1.0, h2c=h2c, ifh2=True)
    g = torch.Generator(device=dev).manual_seed(lx)
    f = c.rhs_assemble(torch.randn(c.n, dtype=torch.float64, device=dev, generator=g))
    return c, f


def jacobi_cg(pkg, c, f, x, steps):
    """(iterates, (p, Ap)) of Jacobi-CG in torch around the library's operator."""
    jac = pkg.api.jacobi_t(c)
    jac.update()
    d, mult, w = jac.dinv(), c.geometry()["mult"], torch.empty_like(f)

    def A(v):
        pkg.ax_helm_t().compute(w, v, c)
        pkg.gs_t(c).op(w)
        pkg.api.bc_list_apply_scalar(c, w)
        return w

    x = x.clone()
    r = f - A(x) if x.any() else f.clone()
    p = d * r
    rz, xs, paps = (r * p * mult).sum(), [], []
    for _ in range(steps):
        pap = (p * A(p) * mult).sum()
        paps.append(float(pap))
        x = x + rz / pap * p
        r = r - rz / pap * w
        new = (r * d * r * mult).sum()
        p, rz = d * r + new / rz * p, new
        xs.append(x)
    return xs, paps


def close(a, b):
    # some hundred roundings of sums of n terms, and four steps whose conditioning is of order 1e3
    return float((a - b).norm()) <= 1e-10 * float(b.norm())


@pytest.mark.parametrize("E,lx", [((3, 2, 1), 2), ((3, 2, 2), 5), ((4, 3, 2), 8), ((2, 2, 2), 10), ((17, 17, 17), 8),
                                  ((28, 28, 27), 5), ((22, 23, 23), 8), ((23, 23, 23), 8)])
def test_jacobi_cg_stopped(pkg, orc, dev, E, lx):
    c, f = plan(pkg, orc, dev, E, lx)
    x0 = T(np.random.default_rng(1).standard_normal(c.n), dev) if c.n < 1e5 else torch.zeros_like(f)
    pkg.gs_t(c).op(x0)
    pkg.api.bc_list_apply_scalar(c, x0)
    ref, _ = jacobi_cg(pkg, c, f, x0, 4)
    ksp = None
    for k in range(1, 5):
        ksp = pkg.krylov_solver_factory(c, "cg", k, 1e-14)
        for again in range(2):  # the same object twice
            x = x0.clone()
            mon = ksp.solve(x, f)
            torch.cuda.synchronize()
            assert mon.iter == k and close(x, ref[k - 1]), (k, again)
        ksp.set_check_every(1)
        x = x0.clone()
        assert ksp.solve(x, f).iter == k and close(x, ref[k - 1])


@pytest.mark.parametrize("E,lx", [((4, 3, 2), 8), ((5, 4, 3), 5)])
def test_breakdown_keeps_the_last_iterate(pkg, orc, dev, E, lx):
    """An indefinite operator: the solve stops at the first direction of
    negative curvature, with the iterate that it came from."""
    for h2c in (-5.0, -20.0, -40.0, -80.0, -160.0, -320.0):
        c, f = plan(pkg, orc, dev, E, lx, h2c)
        x0 = torch.zeros_like(f)
        xs, paps = jacobi_cg(pkg, c, f, x0, 60)
        k = next((i for i, v in enumerate(paps) if v <= 0.0), None)
        if k is not None and k >= 2 and min(abs(v) for v in paps[:k + 1]) > 1e-8 * max(map(abs, paps[:k + 1])):
            break
    else:
        pytest.fail("no operator of the list breaks down after some steps")
    x = x0.clone()
    mon = pkg.krylov_solver_factory(c, "cg", 200, 1e-14).solve(x, f)
    torch.cuda.synchronize()
    assert mon.iter == k and mon.status not in (0, 10), mon
    assert float((x - xs[k - 1]).norm()) <= 1e-7 * float(xs[k - 1].norm())


# just below and above the node count up to which kernels are launched dependently
@pytest.mark.parametrize("E", [(22, 23, 23), (23, 23, 23)])
@pytest.mark.parametrize("fused", [True, False])
def test_schwarz_cg_around_the_dependent_size(pkg, orc, dev, E, fused):
    c, f = plan(pkg, orc, dev, E, 8)
    sw = pkg.schwarz_t(c, coarse=True)
    ref = reference_cg(pkg, c, sw, f, c.geometry()["mult"], None, 3, dev)
    z = [torch.empty(c.n, dtype=torch.float32, device=dev) for _ in range(3)]
    for t in z:
        sw.apply(t, f.float())
    torch.cuda.synchronize()
    assert torch.equal(z[0], z[1]) and torch.equal(z[0], z[2])
    for k in range(1, 4):
        ksp = pkg.krylov_solver_factory(c, "cg_mixed", k, 1e-14)
        ksp.set_inner(1e-12, 1)  # no residual replacement on the way
        ksp.set_schwarz(sw)
        ksp.set_fused_update(fused)
        x = torch.zeros_like(f)
        mon = ksp.solve(x, f)
        torch.cuda.synchronize()
        assert mon.iter == k, mon
        # a step's FP32 roundings are some 1e2 * 2^-24 of its vectors; a missing step moves x by percents
        assert float((x - ref[k - 1]).norm()) <= 1e-4 * float(ref[k - 1].norm()), k
