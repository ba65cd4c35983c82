"""The two-level carry of the dense-Jacobian sweep at the edges of its split.

The chunks' maps are composed in groups, each in slices of 4 * 256 / Dq columns: one
padded size below, at and above each kernel width (Dq = 16, 32, 64, 128), a ragged last
chunk and a ragged last group, and chunk counts with one chunk (no groups), fewer chunks
than a group and several groups.  Accept flags are those of the FP64 sequential chain;
the trajectory is FP32 state with a converged tolerance, 1e-5 of the chain's scale as for
the mode's other tests (the mean norm of its columns: with three coordinates a column can
pass close to the origin, where its own norm says nothing of the rounding that it carries).
"""
import numpy as np
import pytest

import oracle as O
import pmcmc
from pmcmc import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [3, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("T,chunks", [(61, None), (1501, None), (700, "1"), (501, "37"),
                                      (1000, "143"), (2000, "1000")])
def test_groups_match_the_sequential_chain(D, T, chunks, monkeypatch):
    if chunks is not None:
        monkeypatch.setenv("PMCMC_FULL_CHUNKS", chunks)
    rng = np.random.default_rng(1000 * D + T)
    s = 10.0 ** rng.uniform(-1.0, 1.0, D)
    Q = configs.haar_orthogonal(rng, D)
    P = (Q / s) @ Q.T
    P = 0.5 * (P + P.T)
    x0 = rng.standard_normal(D).astype(np.float32)
    sampler = pmcmc.ParallelMALASampler(0.05, T=T, jacobian="full", dtype=np.float32,
                                        tol_abs=1e-7, tol_rel=1e-6, maxiter=200)
    S, info, lp, acc = pmcmc.solve(pmcmc.DensityModel.dense_gaussian(P), sampler, x0, seed=5,
                                   block=2, handle=pmcmc.Handle(0), return_logp=True)
    Xi, u = O.tape(5, 2, D, T)
    ref, acc_ref, _ = O.mala_sequential(O.Target.dense_gauss(P), 0.05, x0.astype(np.float64),
                                        Xi, u)
    assert info["converged"], info
    assert np.array_equal(acc, acc_ref.astype(bool)), np.nonzero(acc != acc_ref)[0][:5]
    S = np.asarray(S, np.float64)
    err = np.max(np.linalg.norm(S - ref, axis=0)) / np.mean(np.linalg.norm(ref, axis=0))
    assert err <= 1e-5
