"""Blocks at the shared-memory bound of the persistent solve keep that path (the target's tables
are left out where they would cost it), and solve as the sequential chain does."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,D,T", [
    (np.float64, 256, 3990), (np.float32, 256, 7000), (np.float32, 256, 7600),
    (np.float32, 200, 10_000), (np.float32, 100, 20_300), (np.float64, 20, 57_271),
    (np.float32, 64, 31_900),
])
def test_block_at_the_bound_stays_persistent(dt, D, T):
    rng = np.random.default_rng(1)
    lam = 10.0 ** rng.uniform(-0.5, 0.5, D)
    x0 = rng.standard_normal(D).astype(dt)
    tol = (1e-7, 1e-6) if dt == np.float32 else (1e-9, 1e-8)
    sampler = pmcmc.ParallelMALASampler(0.03, T=T, jacobian="diag", dtype=dt, tol_abs=tol[0],
                                        tol_rel=tol[1])
    S, info, _, acc = pmcmc.solve(pmcmc.DensityModel.diag_gaussian(lam), sampler, x0, seed=2,
                                  handle=pmcmc.Handle(0), return_logp=True)
    assert info["converged"] and "persistent" in info["path_names"], info
    Xi, u = O.tape(2, 0, D, T)
    R, acc_seq, _ = O.mala_sequential(O.Target.diag_gauss(lam), 0.03, x0.astype(np.float64), Xi, u)
    assert np.array_equal(acc, acc_seq)
    err = np.max(np.linalg.norm(S - R, axis=0) / np.linalg.norm(R, axis=0))
    assert err <= 10 * tol[1]  # what the stopping rule leaves
