"""The forms of the persistent solve's dense columns (P beside the columns or in L2, both products
in one loop or each by itself, one or two CTAs an SM) at the sizes where they change, against the
FP64 sequential chain."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("jac", ["stoch_diag", "diag"])
@pytest.mark.parametrize("dt,D,T", [
    (np.float32, 65, 16), (np.float32, 128, 16),       # above 64 coordinates: a CTA a column
    (np.float32, 106, 300), (np.float32, 110, 300),    # P beside the columns, in L2
    (np.float32, 110, 1300), (np.float32, 129, 1300),  # two CTAs an SM
    (np.float32, 200, 300), (np.float32, 257, 300),
    (np.float64, 65, 16), (np.float64, 129, 200), (np.float64, 257, 100),
    (np.float64, 106, 4200),                           # two CTAs an SM (exact diagonal)
])
def test_dense_forms_match_sequential_chain(h, dt, D, T, jac):
    rng = np.random.default_rng(D)
    Q, R = np.linalg.qr(rng.standard_normal((D, D)))
    P = (Q / 10.0 ** rng.uniform(-0.3, 0.3, D)) @ Q.T
    P = 0.5 * (P + P.T)
    mean = rng.standard_normal(D)
    x0 = (mean + rng.standard_normal(D)).astype(dt)
    eps = 0.3 / D ** (1 / 3)
    model = pmcmc.DensityModel.dense_gaussian(P, mean)
    tol = (1e-7, 1e-6) if dt == np.float32 else (1e-9, 1e-8)
    sampler = pmcmc.ParallelMALASampler(eps, T=T, jacobian=jac, dtype=dt, tol_abs=tol[0],
                                        tol_rel=tol[1], maxiter=1000)
    S, info, _, acc = pmcmc.solve(model, sampler, x0, seed=7, handle=h, return_logp=True)
    assert info["converged"] and "persistent" in info["path_names"], info
    Xi, u = O.tape(7, 0, D, T)
    S_seq, acc_seq, _ = O.mala_sequential(O.Target.dense_gauss(P, mean), eps,
                                          x0.astype(np.float64), Xi, u)
    assert np.array_equal(acc, acc_seq)
    err = np.max(np.linalg.norm(S - S_seq, axis=0) / np.linalg.norm(S_seq, axis=0))
    # the stopping rule leaves tol_rel (1 + the damped sweeps' remainder) of the state
    assert err <= 10 * tol[1]
