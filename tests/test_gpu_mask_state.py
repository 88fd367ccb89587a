"""The Dirichlet mask and what the library derives from it, across the calls
that set the mask aside or change it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

E, R = (4, 3, 2), 0.2


def T(a, dev, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev, dtype)


def masked_plan(pkg, orc, dev, lx):
    c = pkg.coef_t.box(*E, lx, amp=0.05, seed=7, device=dev)
    c.set_mask(T(orc.mask_face_xmax(*E, lx), dev, torch.int32), base=1)
    c.set_coefs(h1c=R * R, h2c=1.0, ifh2=True)
    return c, pkg.schwarz_t(c)


def schwarz_cg(pkg, c, sw):
    ksp = pkg.krylov_solver_factory(c, "cg_mixed", 400, 1e-11)
    ksp.set_schwarz(sw)
    return ksp


def solve(pkg, c, sw, f):
    x = torch.zeros_like(f)
    mon = schwarz_cg(pkg, c, sw).solve(x, c.rhs_assemble(f))
    torch.cuda.synchronize()
    assert mon.status == 0, mon
    return x


def precondition(c, sw, f):
    z = torch.full((c.n,), float("nan"), dtype=torch.float32, device=f.device)
    sw.apply(z, c.rhs_assemble(f).float())
    torch.cuda.synchronize()
    return z


@pytest.mark.parametrize("lx", [4, 6, 8])
@pytest.mark.parametrize("solved_before", [False, True])
def test_filter_leaves_the_mask_as_it_was(pkg, orc, dev, lx, solved_before):
    """The filter runs without the mask and with any solver, the Schwarz-
    preconditioned one included: its result is that of plain CG, and what the
    plan does with its mask afterwards is what a fresh plan does, bit for bit."""
    c, sw = masked_plan(pkg, orc, dev, lx)
    f = T(np.random.default_rng(lx).standard_normal(c.n), dev)
    pkg.gs_t(c).op(f)  # one value per global node
    if solved_before:
        solve(pkg, c, sw, f)
    out, ref = torch.empty_like(f), torch.empty_like(f)
    filt = pkg.PDE_filter_t(c, r=R, abstol=1e-12, max_iter=2000)
    filt.ksp = schwarz_cg(pkg, c, sw)
    assert filt.apply_forward(out, f).status == 0
    c2, _ = masked_plan(pkg, orc, dev, lx)
    c2.set_mask(None)
    assert pkg.PDE_filter_t(c2, r=R, abstol=1e-12, max_iter=2000).apply_forward(ref, f).status == 0
    # both residuals are below 1e-10 of the right-hand side's
    assert float((out - ref).norm()) <= 1e-8 * float(ref.norm())
    c3, sw3 = masked_plan(pkg, orc, dev, lx)
    z = precondition(c3, sw3, f)
    assert not z[torch.from_numpy(orc.mask_face_xmax(*E, lx).astype(np.int64) - 1).to(dev)].any()
    assert torch.equal(precondition(c, sw, f), z)
    assert torch.equal(solve(pkg, c, sw, f), solve(pkg, c3, sw3, f))


@pytest.mark.parametrize("lx", [4, 6, 8])
def test_first_application_under_a_new_mask_is_captured(pkg, orc, dev, lx):
    """The first application after a mask is set allocates nothing: it can be
    recorded into a graph, with the operator and the gather-scatter before it,
    and the replays give what the calls by themselves give."""
    mask = T(orc.mask_face_xmax(*E, lx), dev, torch.int32)
    f = T(np.random.default_rng(lx).standard_normal(24 * lx ** 3), dev, torch.float32)

    def program():
        c = pkg.coef_t.box(*E, lx, amp=0.05, seed=7, device=dev)
        c.set_coefs(h1c=1.0, h2c=0.5, ifh2=True)
        sw = pkg.schwarz_t(c, coarse=True)
        w, z = torch.zeros_like(f), torch.zeros_like(f)

        def run():
            pkg.ax_helm_t().compute(w, f, c)
            pkg.gs_t(c).op(w)
            pkg.api.bc_list_apply_scalar(c, w)
            sw.apply(z, w)

        run()
        c.set_mask(mask, base=1)
        return run, w, z, (c, sw)

    stream = torch.cuda.Stream(dev)
    with torch.cuda.stream(stream):
        run, w_ref, z_ref, keep = program()
        run()
        recorded, w, z, keep2 = program()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        recorded()
    for _ in range(2):
        w.fill_(float("nan"))
        z.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(w, w_ref) and torch.equal(z, z_ref)


@pytest.mark.parametrize("method,bytes_per_node", [("cg", 8), ("cg_mixed", 4)])
def test_first_solve_keeps_weights_of_one_precision(pkg, orc, dev, method, bytes_per_node):
    """What the first Jacobi-preconditioned solve under a mask allocates beyond
    one without: the weights that carry the mask, in its own precision."""
    box, lx = (16, 16, 8), 8

    def allocated(masked):
        c = pkg.coef_t.box(*box, lx, device=dev)
        if masked:
            c.set_mask(T(orc.mask_face_xmax(*box, lx), dev, torch.int32), base=1)
        c.set_coefs(h1c=1.0, h2c=1.0, ifh2=True)
        f = c.rhs_assemble(torch.ones(c.n, dtype=torch.float64, device=dev))
        ksp, x = pkg.krylov_solver_factory(c, method, 3, 1e-14), torch.zeros_like(f)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ksp.solve(x, f)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0], c.n

    (a, n), (b, _) = allocated(True), allocated(False)
    # device memory is handed out in pieces of 2 MiB
    assert abs(a - b - bytes_per_node * n) <= 1 << 21
