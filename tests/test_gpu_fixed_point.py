"""The FP64 contractions evaluated in fixed point (csrc/fx.cuh): every order,
line contents at the edges of the integer range (zeros, subnormals, huge
values, wide ranges within a line, infinities and NaN) and constant factors
inside and outside the range that is folded into the matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def contract(m, D, u, h1):
    """(w, bound): the operator in extended precision and the sum of the absolute values of its terms."""
    Q = np.longdouble
    lx, E = m["lx"], m["E"]
    v = lambda a: np.asarray(a, dtype=Q).reshape(E, lx, lx, lx)
    G = {k: v(m[k]) for k in ("g11", "g12", "g13", "g22", "g23", "g33")}

    def grad(D, U):
        return (np.einsum("il,ekjl->ekji", D, U), np.einsum("jl,ekli->ekji", D, U), np.einsum("kl,elji->ekji", D, U))

    def div(D, a, b, c):
        return (np.einsum("li,ekjl->ekji", D, a) + np.einsum("lj,ekli->ekji", D, b) + np.einsum("lk,elji->ekji", D, c))

    def flux(G, g):
        return (G["g11"] * g[0] + G["g12"] * g[1] + G["g13"] * g[2], G["g12"] * g[0] + G["g22"] * g[1] + G["g23"] * g[2],
                G["g13"] * g[0] + G["g23"] * g[1] + G["g33"] * g[2])

    D = np.asarray(D, dtype=Q)
    w = h1 * div(D, *flux(G, grad(D, v(u))))
    A = {k: abs(g) for k, g in G.items()}
    # each line's terms are held under the line's largest entry
    U = abs(v(u))
    big = lambda ax: np.broadcast_to(U.max(axis=ax, keepdims=True), U.shape)
    a = abs(D)
    g = (np.einsum("il,ekjl->ekji", a, big(3)), np.einsum("jl,ekli->ekji", a, big(2)), np.einsum("kl,elji->ekji", a, big(1)))
    f = flux(A, g)
    top = lambda x, ax: np.broadcast_to(x.max(axis=ax, keepdims=True), x.shape)
    return w.ravel(), (abs(h1) * div(a, top(f[0], 3), top(f[1], 2), top(f[2], 1))).ravel()


def setup(pkg, orc, dev, lx):
    E = (3, 2, 1)
    c = pkg.coef_t.box(*E, lx, amp=0.04, seed=3, device=dev)
    m = {k: t.cpu().numpy() for k, t in c.geometry().items()}
    m.update(lx=lx, E=6, n=6 * lx ** 3)
    return c, m, orc.gll(lx)[2].reshape(lx, lx)


def apply(pkg, c, u, dev):
    w = torch.empty(c.n, dtype=torch.float64, device=dev)
    pkg.ax_helm_t().compute(w, torch.from_numpy(u).to(dev), c)
    torch.cuda.synchronize()
    return w.cpu().numpy()


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("kind", ["random", "wide", "huge", "tiny", "zero_lines"])
@pytest.mark.parametrize("h1", [1.0, -0.01, 3e7])
def test_operator_lines(pkg, orc, dev, lx, kind, h1):
    c, m, D = setup(pkg, orc, dev, lx)
    rng = np.random.default_rng(lx)
    u = rng.standard_normal(m["n"])
    if kind == "wide":
        u *= 10.0 ** rng.uniform(-30, 0, m["n"])
    elif kind == "huge":
        u *= 1e297  # lines beyond the integer form's exponents, results finite
    elif kind == "tiny":
        u *= 1e-290
    elif kind == "zero_lines":
        u.reshape(6, lx, lx, lx)[:, 0] = 0.0
        u.reshape(6, lx, lx, lx)[0] = -0.0
    c.set_coefs(h1c=h1)
    got = apply(pkg, c, u, dev)
    ref, bound = contract(m, D, u, np.longdouble(h1))
    # two contractions of lx terms and the metric products: (4 lx + 16) roundings
    # (the matrix may differ from the library's by one more per entry)
    assert np.all(np.isfinite(got))
    assert np.all(abs(got.astype(np.longdouble) - ref) <= (4 * lx + 16) * EPS * bound + np.longdouble(5e-324) * 64)
    if kind == "zero_lines":
        assert not got.reshape(6, -1)[0].any()  # an element of zeros stays exactly zero


@pytest.mark.parametrize("lx", [2, 5, 8])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_operator_passes_non_finite_on(pkg, orc, dev, lx, bad):
    """NaN and infinity reach exactly the nodes the plain FP64 sums give them
    to: the planes through their node, in their own element."""
    c, m, D = setup(pkg, orc, dev, lx)
    c.set_coefs(h1c=1.0)
    u = np.random.default_rng(1).standard_normal(m["n"])
    i, j, k = 0, 1, lx - 1
    u.reshape(6, lx, lx, lx)[4, k, j, i] = bad
    got = apply(pkg, c, u, dev).reshape(6, lx, lx, lx)
    hit = np.zeros(got.shape, dtype=bool)
    hit[4, k], hit[4, :, j], hit[4, :, :, i] = True, True, True
    assert np.array_equal(~np.isfinite(got), hit)
    u.reshape(6, lx, lx, lx)[4, k, j, i] = 0.0
    assert np.array_equal(got[~hit], apply(pkg, c, u, dev).reshape(got.shape)[~hit])


@pytest.mark.parametrize("lx", [4, 5, 6, 7, 8])
@pytest.mark.parametrize("mode", ["adjoint", "linear"])
def test_dealias_edges(pkg, orc, dev, lx, mode):
    """Element counts off the block's size, zero velocities, and a NaN that stays in its element."""
    E = (5, 1, 1)
    c = pkg.coef_t.box(*E, lx, amp=0.03, seed=3, device=dev)
    adv = pkg.adv_lin_dealias_t(c)
    run = adv.compute_adjoint if mode == "adjoint" else adv.compute_linear
    g = torch.Generator(device=dev).manual_seed(lx)
    F = lambda: torch.randn(c.n, dtype=torch.float64, device=dev, generator=g)
    u, b, f = [F() for _ in range(3)], [F() for _ in range(3)], [F() for _ in range(3)]
    z = [torch.zeros_like(f[0]) for _ in range(3)]
    out = [t.clone() for t in f]
    run(*u, *z, *out)
    assert all(torch.equal(a, q) for a, q in zip(out, f))  # no base flow: nothing to add
    clean = [t.clone() for t in f]
    run(*u, *b, *clean)
    u[1].view(5, -1)[2, 3] = float("nan")
    out = [t.clone() for t in f]
    run(*u, *b, *out)
    for a, q in zip(out, clean):
        a, q = a.view(5, -1), q.view(5, -1)
        assert torch.isnan(a[2]).all()
        assert torch.equal(a[[0, 1, 3, 4]], q[[0, 1, 3, 4]])
