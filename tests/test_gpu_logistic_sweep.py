"""The kernels after the tensor-core passes of a sweep: near-tie decisions in FP64 (with more
candidates than one refinement takes, too) and the scan over several launches, checked at
the returned trajectory against log alpha in NumPy FP64."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


def _log_alpha(X, y, eps, Xb, xi):
    """log alpha of every step from the columns of Xb (D, T), FP64."""
    def model(B):
        L = X @ B
        lp = y @ L - np.logaddexp(0, L).sum(0) - 0.5 * (B * B).sum(0)
        return lp, X.T @ (y[:, None] - 1 / (1 + np.exp(-L))) - B
    lx, gx = model(Xb)
    Y = Xb + eps * gx + np.sqrt(2 * eps) * xi
    ly, gy = model(Y)
    r = Xb - Y - eps * gy
    return ly - lx - (r * r).sum(0) / (4 * eps) + 0.5 * (xi * xi).sum(0)


@pytest.mark.parametrize("N,D,T", [
    (12, 3, 400_000),   # about 400 candidates for 256 places; four launches of the scan
    (300, 40, 3001), (2000, 129, 2500), (700, 300, 2000),
    (9, 512, 300),      # fewer rows than an MMA's tile pair, the most coordinates
])
def test_decisions_follow_fp64_log_alpha(h, N, D, T):
    rng = np.random.default_rng(N + T)
    X = (rng.standard_normal((N, D)) / np.sqrt(D)).astype(np.float32).astype(np.float64)
    y = (rng.random(N) < 1 / (1 + np.exp(-X @ rng.standard_normal(D)))).astype(np.float64)
    eps = 0.1 / (1 + 0.25 * N / D)
    model = pmcmc.DensityModel.logistic(X, y)
    sampler = pmcmc.ParallelMALASampler(eps, T=T, dtype=np.float32, maxiter=400)
    S, info, lp, acc = pmcmc.solve(model, sampler, np.zeros(D, np.float32), seed=4, handle=h,
                                   return_logp=True)
    assert info["converged"] and info["path"] & 64, info
    Xi, u = O.tape(4, 0, D, T)
    xb = np.concatenate([np.zeros((D, 1)), np.asarray(S, np.float64)[:, :-1]], axis=1)
    m = _log_alpha(X, y, eps, xb, Xi.astype(np.float64)) - np.log(u.astype(np.float64))
    assert np.array_equal(acc, m > 0)
    # near ties (within 1e-3; a quarter of that with more than 256 of them) are decided in
    # FP64, sums of N terms of about 1; the smallest margin is one here
    assert np.abs(m).min() < (1e-3 if np.sum(np.abs(m) < 1e-3) <= 256 else 2.5e-4)
    assert abs(info["min_margin"] - np.abs(m).min()) <= 1e-11 * (1 + N)
    # the recursion holds at the returned state to the stopping rule (1e-6 + 1e-5 |S|)
    assert info["max_defect"] <= 1e-5 * (1 + np.abs(S).max())
