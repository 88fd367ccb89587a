"""Derivatives and the FP64 operator node by node: the rounding of a result is
bounded by the terms of its own sum, also where one entry of a line is larger
than all others and meets a zero of the matrix."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

Q = np.longdouble
EPS = Q(2.0) ** -53
E = (3, 2, 2)


def fields(lx, kind, rng):
    """Normal values, of one order, with outliers, or over many orders; one node per element."""
    n = 12 * lx ** 3
    u = rng.standard_normal(n)
    if kind == "spikes":
        u *= np.where(rng.random(n) < 0.5 / lx, 2.0 ** rng.uniform(0, 45, n), 1.0)
    elif kind == "wide":
        u *= 10.0 ** rng.uniform(-12, 0, n)
    elif kind == "one":
        v = np.zeros((12, lx, lx, lx))
        for e in range(12):
            v[(e,) + tuple(rng.integers(0, lx, 3))] = rng.standard_normal()
        u = v.ravel()
    return u


def grad(D, u):
    return np.einsum("il,ekjl->ekji", D, u), np.einsum("jl,ekli->ekji", D, u), np.einsum("kl,elji->ekji", D, u)


def div(D, f):
    return (np.einsum("li,ekjl->ekji", D, f[0]) + np.einsum("lj,ekli->ekji", D, f[1])
            + np.einsum("lk,elji->ekji", D, f[2]))


@pytest.fixture(scope="module")
def mesh(pkg, orc, dev):
    made = {}

    def get(lx):
        if lx not in made:
            c = pkg.coef_t.box(*E, lx, amp=0.04, seed=3, device=dev).metrics()
            D = orc.gll(lx)[2].reshape(lx, lx).astype(Q)
            D[np.arange(1, lx - 1), np.arange(1, lx - 1)] = 0  # as the nodes' symmetry has it
            made[lx] = c, D, orc.gll(lx)[1].astype(Q)
        return made[lx]

    return get


# Bounds in units of 2^-53 times the terms of the sum: lx for a sum in any
# order; 480 for a sum of integers, whose error is half of one such unit of the
# row's largest entry times the line's largest, when that is less than eight
# times the next (or the sum is not one of integers) and the smallest
# off-diagonal entry of D^T at least 1/120 of its row's largest; 8 for D itself.
def tol(lx):
    return (lx + 480 + 8) * EPS


def cofactors(D, X):
    (xr, xs, xt), (yr, ys, yt), (zr, zs, zt) = (grad(D, a) for a in X)
    m = [ys * zt - yt * zs, xt * zs - xs * zt, xs * yt - xt * ys, yt * zr - yr * zt, xr * zt - xt * zr,
         xt * yr - xr * yt, yr * zs - ys * zr, xs * zr - xr * zs, xr * ys - xs * yr]
    return m, max(abs(v).max() for v in m)


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("kind", ["normal", "spikes", "wide", "one"])
def test_gradient(pkg, mesh, dev, lx, kind):
    c, D, w = mesh(lx)
    w3 = w[:, None, None] * w[None, :, None] * w[None, None, :]
    X = [t.cpu().numpy().astype(Q).reshape(12, lx, lx, lx) for t in (c.x, c.y, c.z)]
    m, top = cofactors(D, X)
    u = fields(lx, kind, np.random.default_rng(lx))
    U = u.astype(Q).reshape(12, lx, lx, lx)
    ud, g, a = torch.from_numpy(u).to(dev), grad(D, U), grad(abs(D), abs(U))
    out = [torch.empty_like(ud) for _ in range(3)]
    pkg.api.opgrad(*out, ud, c)
    for k in range(3):
        ref = w3 * sum(m[3 * d + k] * g[d] for d in range(3))
        size = w3 * top * sum(a)
        err = abs(out[k].cpu().numpy().astype(Q).reshape(ref.shape) - ref)
        # a cofactor's own rounding: two sums of lx terms, |D| |x| some 300 times a derivative of x at lx 10
        assert np.all(err <= (tol(lx) + 3000 * EPS) * size), (k, float((err / (size + Q(1e-4000))).max() / EPS))


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("kind", ["spikes", "wide", "one"])
def test_transposed_gradient(pkg, mesh, dev, lx, kind):
    c, D, w = mesh(lx)
    w3 = w[:, None, None] * w[None, :, None] * w[None, None, :]
    X = [t.cpu().numpy().astype(Q).reshape(12, lx, lx, lx) for t in (c.x, c.y, c.z)]
    m, top = cofactors(D, X)
    u = fields(lx, kind, np.random.default_rng(lx))
    U = w3 * u.astype(Q).reshape(12, lx, lx, lx)
    ud, out = torch.from_numpy(u).to(dev), torch.empty(c.n, dtype=torch.float64, device=dev)
    for k in range(3):
        pkg.api.cdtp(out, ud, k, c)
        ref = div(D, [m[3 * d + k] * U for d in range(3)])
        size = top * div(abs(D), [abs(U)] * 3)
        err = abs(out.cpu().numpy().astype(Q).reshape(ref.shape) - ref)
        assert np.all(err <= (tol(lx) + 3000 * EPS) * size), (k, float((err / (size + Q(1e-4000))).max() / EPS))


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("kind", ["normal", "spikes", "wide", "one", "h1"])
def test_operator(pkg, mesh, dev, lx, kind):
    c, D, _ = mesh(lx)
    rng = np.random.default_rng(lx)
    G = {k: t.cpu().numpy().astype(Q).reshape(12, lx, lx, lx) for k, t in c.geometry().items()}
    u = fields(lx, kind, rng)
    U = u.astype(Q).reshape(12, lx, lx, lx)
    h1 = np.where(rng.random(c.n) < 0.5 / lx, 2.0 ** rng.uniform(0, 45, c.n), 1.0) if kind == "h1" else np.ones(c.n)
    c.set_coefs(h1=torch.from_numpy(h1).to(dev) if kind == "h1" else None, h1c=1.0)
    H = h1.astype(Q).reshape(U.shape)
    w = torch.empty(c.n, dtype=torch.float64, device=dev)
    pkg.ax_helm_t().compute(w, torch.from_numpy(u).to(dev), c)

    def flux(G, g):
        return (H * (G["g11"] * g[0] + G["g12"] * g[1] + G["g13"] * g[2]),
                H * (G["g12"] * g[0] + G["g22"] * g[1] + G["g23"] * g[2]),
                H * (G["g13"] * g[0] + G["g23"] * g[1] + G["g33"] * g[2]))

    ref = div(D, flux(G, grad(D, U)))
    A = {k: abs(v) for k, v in G.items()}
    size = div(abs(D), flux(A, grad(abs(D), abs(U))))
    err = abs(w.cpu().numpy().astype(Q).reshape(ref.shape) - ref)
    # two sums and four metric products
    assert np.all(err <= (2 * tol(lx) + 8 * EPS) * size), float((err / (size + Q(1e-4000))).max() / EPS)
