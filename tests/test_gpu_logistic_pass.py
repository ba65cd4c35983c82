"""The tensor-core pass at the edges of its tiles (64 columns, 64 rows, 128 / 256 / 512 values
of d, rows split over CTAs): a solve against the FP64 sequential chain on the same tape."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("N,D,T", [
    (1, 1, 1), (63, 4, 63), (64, 5, 64), (65, 127, 65),  # one block, one tile; one past them
    (128, 128, 129), (129, 129, 128), (300, 250, 40),    # an even and an odd number of blocks
    (1500, 256, 70),                                     # rows split over CTAs, two boxes of d
    (700, 16, 9500),                                     # more tiles than SMs, no split
    (65, 257, 63), (64, 384, 129), (1000, 512, 65),      # two CTAs a tile, each half of d
])
def test_pass_edges(h, N, D, T):
    rng = np.random.default_rng(N + D + T)
    X = (rng.standard_normal((N, D)) / np.sqrt(D)).astype(np.float32).astype(np.float64)
    y = (rng.random(N) < 1 / (1 + np.exp(-X @ rng.standard_normal(D)))).astype(np.float64)
    eps = 0.1 / (1 + 0.25 * N / D)
    model = pmcmc.DensityModel.logistic(X, y)
    # the iterate stops within about 1e-7 + 1e-6 |S| of the chain
    sampler = pmcmc.ParallelMALASampler(eps, T=T, dtype=np.float32, tol_abs=1e-7, tol_rel=1e-6,
                                        maxiter=400)
    S, info, lp, acc = pmcmc.solve(model, sampler, np.zeros(D, np.float32), seed=6, handle=h,
                                   return_logp=True)
    tg = O.Target.logistic(X, y)
    Xi, u = O.tape(6, 0, D, T)
    R, racc, _ = O.mala_sequential(tg, eps, np.zeros(D), Xi, u)
    assert info["converged"] and info["path"] & 8, info
    assert np.array_equal(acc, racc)
    scale = max(1.0, np.abs(R).max())
    assert np.abs(S - R).max() <= 1e-5 * scale
    # the log density at the returned state: N terms rounded to FP32, and the state's rounding
    step = max(1, T // 50)
    ref = np.array([O.logp(tg, np.asarray(S[:, t], np.float64)) for t in range(0, T, step)])
    np.testing.assert_allclose(lp[::step], ref, rtol=1e-6, atol=1e-5 * np.sqrt(N))
