"""The element-tile kernels where a block takes several groups of elements one
after another, the last of them short: the results of a mesh of thousands of
elements are, bit for bit, those of the same elements as small meshes, of which
every block has one group."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def counts(lx):  # elements, elements of a piece
    return (40009, 997) if lx <= 3 else (5003, 97)


def terms(pkg, c, F):
    """Every element-local result for the fields F on the mesh c (no shared nodes)."""
    A, lx = pkg.api, c.lx
    out = []

    def new(k):
        t = [torch.zeros(c.n, dtype=torch.float64, device=F[0].device) for _ in range(k)]
        out.extend(t)
        return t

    A.dudxyz(*new(1), F[0], "y", c)
    A.opgrad(*new(3), F[0], c)
    A.cdtp(*new(1), F[0], "z", c)
    A.conv1(*new(1), F[0], F[1], F[2], F[3], c)
    A.curl(*new(3), F[1], F[2], F[3], c)
    for adv in [pkg.adv_lin_no_dealias_t(c)] + ([pkg.adv_lin_dealias_t(c)] if lx in (4, 5, 6, 7, 8) else []):
        adv.compute_adjoint(*F[1:4], *F[4:7], *new(3))
        adv.compute_linear(*F[1:4], *F[4:7], *new(3))
    f = new(3)
    A.adjoint_minimum_dissipation_source_term_t(f, *F[1:4], c, obj_scale=0.5).compute()
    for mu in (0.01, F[7]):
        pkg.pnpn_prs_res_t().compute(F[0], *new(1), *F[1:4], *F[4:7], *F[1:4], c, mu=mu, rho=1.5)
        pkg.pnpn_vel_res_t().compute(*F[1:4], *new(3), F[0], *F[4:7], c, mu=mu, rho=1.5, bd=1.5, dt=1e-2)
    for h1 in (None, F[7]):
        c.set_coefs(h1=h1, h1c=0.7, h2=F[7], ifh2=True)
        pkg.ax_helm_t().compute(*new(1), F[0], c)
        jac = A.jacobi_t(c)
        jac.update()
        out.append(jac.dinv().clone())
        w = torch.zeros(c.n, dtype=torch.float32, device=F[0].device)
        pkg.ax_helm_t().compute(w, F[0].float(), c)
        out.append(w)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("lx", [2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_large_mesh_equals_its_pieces(pkg, dev, lx):
    # off every group size, and more groups than blocks run at a time on 152 SMs
    L, (N, PIECE) = lx ** 3, counts(lx)
    x, y, z, _ = pkg.api.build_box(N, 1, 1, lx, hi=(float(N), 1.0, 1.0), amp=0.04, seed=lx, device=dev)
    gid = torch.arange(N * L, device=dev)
    g = torch.Generator(device=dev).manual_seed(lx)
    F = [torch.randn(N * L, dtype=torch.float64, device=dev, generator=g) for _ in range(7)]
    F.append(torch.rand(N * L, dtype=torch.float64, device=dev, generator=g) + 0.5)
    whole = terms(pkg, pkg.coef_t(N, lx, x, y, z, gid), F)
    for e in range(0, N, PIECE):
        s = slice(e * L, min(N, e + PIECE) * L)
        part = terms(pkg, pkg.coef_t(min(N, e + PIECE) - e, lx, x[s].clone(), y[s].clone(), z[s].clone(),
                                     torch.arange(s.stop - s.start, device=dev)), [t[s].clone() for t in F])
        for k, (a, b) in enumerate(zip(whole, part)):
            assert torch.equal(a[s], b), (e, k)
