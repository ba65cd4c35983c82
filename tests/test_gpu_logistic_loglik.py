"""Log-likelihood of the tensor-core pass where the rows are well separated: every row adds
log(1 + exp(-|l|)), down to 4e-8 each, and the sum keeps its relative accuracy."""
import numpy as np
import pytest

import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("N,D", [(10_000, 24), (10_001, 200), (4000, 400)])
@pytest.mark.parametrize("scale", [1.0, 6.0, 12.0, 17.0])
def test_loglik_keeps_small_terms(h, N, D, scale):
    rng = np.random.default_rng(N + D)
    side = np.where(rng.random(N) < 0.5, -1.0, 1.0)
    X = side[:, None] * scale / D * rng.uniform(0.9, 1.1, (N, D))  # logits about +- scale at x = 1
    tau = 1e-12
    model = pmcmc.DensityModel.logistic(X, (side > 0).astype(float), tau)
    sampler = pmcmc.ParallelMALASampler(1e-10, T=70, dtype=np.float32)
    S, info, lp, _ = pmcmc.solve(model, sampler, np.ones(D, np.float32), seed=1, handle=h,
                                 return_logp=True)
    assert info["converged"] and "tensor_core" in info["path_names"]
    S = np.asarray(S, np.float64)
    l = X @ S
    exact = -np.log1p(np.exp(-side[:, None] * l)).sum(0) - 0.5 * tau * (S * S).sum(0)
    # a logit is off by the operands' 2^-21 and the FP32 accumulation of D / 16 + 4 steps, its
    # exponential by the rounding of l log2(e) and 2 ulp, log(1 + e) by 1e-6, the result by 2^-24
    tol = scale * 1.1 * (2.0 ** -21 + (D / 16 + 4) * 2.0 ** -23 + 2.0 ** -22) + 2e-6
    np.testing.assert_allclose(np.asarray(lp, np.float64), exact, rtol=tol)
