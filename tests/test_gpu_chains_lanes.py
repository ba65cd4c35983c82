"""The register-resident diagonal chain kernel at the edges of its lane layout: one
coordinate, a full and a ragged last quad, steps drawn 32 / nq at a time (32, 6, 4, 1), the
lanes of one, two and four coordinates, the largest D of the kernel and the
first above it, lengths around the 32-step batches, and one or several chains a CTA.
FP64 chains against the sequential oracle, 1e-12 (the bar of the mode's other tests:
the arithmetic is FP64 and a chain's rounding grows by its length, at most 70 steps here).
"""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 4, 20, 31, 32, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("T,n", [(1, 1), (32, 3), (70, 300)])
def test_diag_chains_match_the_sequential_oracle(D, T, n):
    rng = np.random.default_rng(100 * D + T)
    lam, mean = 10 ** rng.uniform(-1, 0.5, D), rng.standard_normal(D)
    model = pmcmc.DensityModel.diag_gaussian(lam, mean=mean)
    eps = 0.3 / lam.max() / D ** (1 / 3)
    x0 = mean + rng.standard_normal((n, D))
    seeds = [int(s) for s in rng.integers(1, 1 << 40, n)]
    S, lp, acc = pmcmc.mala_chains(model, pmcmc.ParallelMALASampler(eps, T=T), x0, seeds, block=1)
    tg = O.Target.diag_gauss(lam, mean)
    for c in sorted({0, n // 2, n - 1}):
        Xi, u = O.tape(seeds[c], 1, D, T)
        ref, acc_ref, _ = O.mala_sequential(tg, eps, x0[c], Xi, u)
        assert np.array_equal(acc[c], acc_ref), c
        np.testing.assert_allclose(S[c].T, ref, rtol=1e-12, atol=1e-12)
        np.testing.assert_allclose(lp[c], [O.logp(tg, ref[:, t]) for t in range(T)],
                                   rtol=1e-12, atol=1e-12 * D)
