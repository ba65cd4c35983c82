"""The sweep's scan in one CTA (runs of at most 32 columns) and, one column later, over the
grid: the accept flags are those of the FP64 log alpha at the returned state, and the
recursion holds there to the stopping rule (1e-6 + 1e-5 |S|), as in the sweep's other test.
"""
import numpy as np
import pytest

import oracle as O
import pmcmc

from test_gpu_logistic_sweep import _log_alpha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damping", [1.0, 0.8])
@pytest.mark.parametrize("D,T", [(3, 1), (3, 2048), (3, 2049), (24, 320), (24, 321), (100, 64),
                                 (100, 65), (256, 32), (256, 33)])
def test_one_cta_scan(D, T, damping):
    N = 150
    rng = np.random.default_rng(D + T)
    X = (rng.standard_normal((N, D)) / np.sqrt(D)).astype(np.float32).astype(np.float64)
    y = (rng.random(N) < 1 / (1 + np.exp(-X @ rng.standard_normal(D)))).astype(np.float64)
    eps = 0.1 / (1 + 0.25 * N / D)
    sampler = pmcmc.ParallelMALASampler(eps, T=T, dtype=np.float32, maxiter=800, damping=damping)
    S, info, lp, acc = pmcmc.solve(pmcmc.DensityModel.logistic(X, y), sampler,
                                   np.zeros(D, np.float32), seed=4, handle=pmcmc.Handle(0),
                                   return_logp=True)
    assert info["converged"] and info["path"] & 64, info
    Xi, u = O.tape(4, 0, D, T)
    xb = np.concatenate([np.zeros((D, 1)), np.asarray(S, np.float64)[:, :-1]], axis=1)
    m = _log_alpha(X, y, eps, xb, Xi.astype(np.float64)) - np.log(u.astype(np.float64))
    assert np.array_equal(acc, m > 0)
    assert info["max_defect"] <= 1e-5 * (1 + np.abs(S).max())
