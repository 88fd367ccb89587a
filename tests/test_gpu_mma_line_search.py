"""The interior-point line search where it takes something else than its first
trial: none at all, and one that comes after rejected ones."""
import numpy as np
import pytest
import torch

from oracle.mma_ref import MMA

pytestmark = pytest.mark.gpu


def T(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)


def problem(n, m):
    rng = np.random.default_rng(n + m)
    w, V = rng.uniform(0.5, 2.0, n), rng.uniform(0.1, 1.0, (m, n))
    lim = 0.4 * V.mean(axis=1)
    return lambda x: (-w / x ** 2 / n, (V * x).mean(axis=1) - lim, V / n)


@pytest.mark.parametrize("n", [5, 301])  # nine and eight levels of the interior-point parameter
@pytest.mark.parametrize("m", [1, 3])
@pytest.mark.parametrize("bad", ["value", "gradient"])
@pytest.mark.parametrize("updates_before", [0, 2])
@pytest.mark.parametrize("max_iter", [1, 2, 3, 100])
def test_non_finite_data_leave_the_starting_point(pkg, dev, n, m, bad, updates_before, max_iter):
    """With a residual that is not finite no trial is taken, whatever the
    number of Newton steps: the subproblem's starting point is the design, the
    middle of the move limits, as in the reference's algorithm."""
    prob, x0 = problem(n, m), np.full(n, 0.5)
    ref = MMA(x0, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0)
    xd, xr = T(x0, dev), x0.copy()
    opt = pkg.mma_t(xd, n, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0, max_iter=100 if updates_before else max_iter)
    for it in range(1, updates_before + 1):
        df0, f, df = prob(xd.cpu().numpy())
        opt.update(it, xd, T(df0, dev), f, T(df.T.ravel(), dev))
        df0, f, df = prob(xr)
        xr = ref.update(it, xr, df0, f, df)
    x = xd.cpu().numpy()
    df0, f, df = prob(x)
    if bad == "value":
        f = f.copy()
        f[0] = np.nan
    else:
        df0 = df0.copy()
        df0[3] = np.inf
    trials = opt.counts[1]
    opt.update(updates_before + 1, xd, T(df0, dev), f, T(df.T.ravel(), dev))
    with np.errstate(invalid="ignore"):
        ref.gensub(updates_before + 1, x, df0, f, df)
    assert opt.counts[1] == trials
    # the asymptotes of both come from iterates that agree to 1e-8
    assert np.allclose(xd.cpu().numpy(), 0.5 * (ref.alpha + ref.beta), rtol=1e-7, atol=0)


@pytest.mark.parametrize("m", [1, 3])
def test_rejected_trials(pkg, dev, m):
    n, its = 5, 6
    prob, x0 = problem(n, m), np.full(n, 0.5)
    ref = MMA(x0, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0)
    xd, xr = T(x0, dev), x0.copy()
    opt = pkg.mma_t(xd, n, m, 1.0, 0.0, 100.0, 1.0, 0.01, 1.0)
    for it in range(1, its + 1):
        df0, f, df = prob(xd.cpu().numpy())
        opt.update(it, xd, T(df0, dev), f, T(df.T.ravel(), dev))
        df0, f, df = prob(xr)
        xr = ref.update(it, xr, df0, f, df)
        # rounding of the Newton systems, condition some 1e4
        assert np.allclose(xd.cpu().numpy(), xr, rtol=1e-8, atol=1e-10)
    steps, trials, _ = opt.counts
    assert trials > steps and steps == ref.newton_steps
