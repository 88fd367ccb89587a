"""The Jacobi diagonal where the coefficient jumps inside elements: every node's
value is as good as the terms of its own sum allow."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

Q = np.longdouble


@pytest.mark.parametrize("lx", range(2, 11))
@pytest.mark.parametrize("kind", ["log", "jumps"])
def test_diagonal(pkg, orc, dev, lx, kind):
    E = (3, 2, 2)
    c = pkg.coef_t.box(*E, lx, amp=0.04, seed=3, device=dev)
    rng = np.random.default_rng(lx)
    h1 = 10.0 ** rng.uniform(-12, 0, c.n) if kind == "log" else np.where(rng.random(c.n) < 0.7, 1e-9, 1.0)
    c.set_coefs(h1=torch.from_numpy(h1).to(dev))
    jac = pkg.api.jacobi_t(c)
    jac.update()
    G = {k: t.cpu().numpy().astype(Q).reshape(12, lx, lx, lx) for k, t in c.geometry().items()}
    D = orc.gll(lx)[2].reshape(lx, lx).astype(Q)
    D[np.arange(1, lx - 1), np.arange(1, lx - 1)] = 0  # as the nodes' symmetry has it
    D2, d = D * D, np.diag(D)
    h = h1.astype(Q).reshape(12, lx, lx, lx)
    main = (np.einsum("li,ekjl->ekji", D2, h * G["g11"]) + np.einsum("lj,ekli->ekji", D2, h * G["g22"])
            + np.einsum("lk,elji->ekji", D2, h * G["g33"]))
    i, j, k = d[None, None, None, :], d[None, None, :, None], d[None, :, None, None]
    cross = [2 * h * i * j * G["g12"], 2 * h * i * k * G["g13"], 2 * h * j * k * G["g23"]]
    ids = np.unique(c.gid.cpu().numpy(), return_inverse=True)[1].ravel()

    def assembled(v):
        t = np.zeros(ids.max() + 1, dtype=Q)
        np.add.at(t, ids, v.ravel())
        return t[ids]

    diag, size = assembled(main + sum(cross)), assembled(main + sum(map(abs, cross)))
    got = jac.dinv().cpu().numpy().astype(Q)
    # D within 8 roundings an entry (squared: 16), products and 3 lx + 4 terms, the assembly, the reciprocal
    assert np.all(abs(got * diag - 1) <= (3 * lx + 40) * Q(2.0) ** -53 * size / diag)
