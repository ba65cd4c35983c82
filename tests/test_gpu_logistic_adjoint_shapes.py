"""The adjoint's Hessian-vector products at the edges of their tiles: coordinates around 8
(one tile), 64 and 128 (one and two tiles a warp; 132 takes the products by GEMM), rows
around the chunk of 64, fewer rows than coordinates (one split), columns around the tile of
32.  Against the dense FP64 restatement at the same trajectory, 1e-8 relative: the iterations
stop at 1e-12 of lambda's maximum and everything is FP64.
"""
import numpy as np
import pytest

import np_oracle as NO
import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("objective", ["esjd", "mean_sq"])
@pytest.mark.parametrize("N,D,T", [(5, 3, 2), (64, 8, 33), (65, 9, 32), (300, 12, 70),
                                   (129, 63, 64), (700, 64, 97), (100, 65, 40), (640, 100, 31),
                                   (63, 127, 33), (400, 128, 34), (200, 132, 33)])
def test_adjoint_matches_the_restatement(N, D, T, objective):
    rng = np.random.default_rng(N + D + T)
    X = (rng.standard_normal((N, D)) / np.sqrt(D)).astype(np.float32).astype(np.float64)
    y = (rng.random(N) < 1 / (1 + np.exp(-X @ rng.standard_normal(D)))).astype(np.float64)
    eps = 0.05
    model = pmcmc.DensityModel.logistic(X, y)
    sampler = pmcmc.ParallelMALASampler(eps, T=T, dtype=np.float64, tol_abs=1e-12,
                                        tol_rel=1e-10, maxiter=400)
    x0 = rng.standard_normal(D) * 0.3
    h = pmcmc.Handle(0)
    S, info = pmcmc.solve(model, sampler, x0, seed=8, block=1, handle=h)
    assert info["converged"]
    g = pmcmc.adjoint(model, sampler, x0, S, objective=objective, seed=8, block=1, handle=h)
    Xi, u = O.tape(8, 1, D, T)
    ref = NO.logistic_adjoint(X, y, eps, x0, Xi, u, np.asarray(S), objective)
    assert abs(g["d_epsilon"] - ref) <= 1e-8 * abs(ref)
