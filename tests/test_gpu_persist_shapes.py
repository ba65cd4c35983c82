"""The persistent solve over its shapes: lanes a column (1 .. 32, D at each edge), one CTA or many,
runs of the in-CTA scan, shares of the dense products, staged and piped host outputs -- against
the FP64 sequential chain on the same tape."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


def _problem(kind, D, seed):
    rng = np.random.default_rng(seed)
    mean = rng.standard_normal(D)
    if kind == "diag":
        lam = 10.0 ** rng.uniform(-0.5, 0.5, D)
        return pmcmc.DensityModel.diag_gaussian(lam, mean=mean), O.Target.diag_gauss(lam, mean)
    A = rng.standard_normal((D, D)) / np.sqrt(D)
    P = A @ A.T + 0.5 * np.eye(D)
    P = 0.5 * (P + P.T)
    return pmcmc.DensityModel.dense_gaussian(P, mean=mean), O.Target.dense_gauss(P, mean)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind,jac,D,T", [
    ("diag", "diag", 1, 1), ("diag", "diag", 4, 256), ("diag", "stoch_diag", 4, 257),
    ("diag", "diag", 5, 255), ("diag", "stoch_diag", 8, 300), ("diag", "diag", 9, 128),
    ("diag", "stoch_diag", 16, 129), ("diag", "diag", 17, 64), ("diag", "stoch_diag", 32, 65),
    ("diag", "diag", 33, 32), ("diag", "stoch_diag", 64, 700), ("diag", "diag", 65, 33),
    ("diag", "diag", 128, 1000), ("diag", "diag", 129, 50), ("diag", "diag", 257, 90),
    ("diag", "stoch_diag", 300, 40),
    ("dense", "stoch_diag", 3, 16), ("dense", "diag", 32, 17), ("dense", "stoch_diag", 33, 200),
    ("dense", "diag", 64, 40), ("dense", "stoch_diag", 65, 150), ("dense", "diag", 130, 20),
])
def test_persist_shapes(h, dt, kind, jac, D, T):
    model, tg = _problem(kind, D, D + T)
    eps = 0.1
    # the iterate stops within tol_abs + tol_rel |S| of the chain
    rel = 1e-6 if dt == np.float32 else 1e-11
    s = pmcmc.ParallelMALASampler(eps, T=T, jacobian=jac, dtype=dt, tol_abs=rel, tol_rel=rel,
                                  maxiter=2000)
    x0 = np.random.default_rng(1).standard_normal(D).astype(dt)
    S, info, lp, acc = pmcmc.solve(model, s, x0, seed=3, handle=h, return_logp=True)
    assert info["converged"] and info["path"] & 32, info
    Xi, u = O.tape(3, 0, D, T)
    R, racc, _ = O.mala_sequential(tg, eps, x0.astype(np.float64), Xi, u)
    assert np.array_equal(acc, racc)
    scale = max(1.0, np.abs(R).max())
    assert np.abs(S - R).max() <= 10 * rel * scale
    ref = np.array([O.logp(tg, np.asarray(S[:, t], np.float64)) for t in range(T)])
    np.testing.assert_allclose(lp, ref, rtol=1e-6 if dt == np.float32 else 1e-12, atol=1e-12)


@pytest.mark.parametrize("D,T,N", [(2, 64, 500), (3, 50, 50 * 4), (40, 700, 30_000)])
def test_host_blocks_equal_device_blocks(h, D, T, N):
    """One launch with staged outputs (below 4 MB), or a launch and a copy a block: the same
    bits as one launch into device memory."""
    torch = pytest.importorskip("torch")
    model, _ = _problem("diag", D, 5)
    s = pmcmc.ParallelMALASampler(0.1, T=T, jacobian="diag", dtype=np.float32)
    x0 = np.zeros(D, np.float32)
    a = pmcmc.sample(model, s, N, seed=9, initial_params=x0, handle=h)
    b = pmcmc.sample(model, s, N, seed=9, initial_params=torch.from_numpy(x0).cuda(), handle=h)
    assert np.array_equal(a.values, b.values.cpu().numpy())
    assert np.array_equal(a.logp, b.logp.cpu().numpy())
    assert np.array_equal(a.accepted, b.accepted.cpu().numpy())
    assert a.info["iters"] == b.info["iters"] and a.info["n_accept"] == b.info["n_accept"]
