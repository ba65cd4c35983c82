"""Bounded device waits of the grid barrier (persistent solve, scans, near ties) and of the
two-CTA pass's mailbox: each gives up at its bound and returns PMCMC_ERR_TIMEOUT, and the same
handle, whose barrier word the first has left mid-phase, then solves as before."""
import numpy as np
import pytest

import pmcmc
from pmcmc import _lib as L

pytestmark = pytest.mark.gpu


def _solves(h):
    """A persistent solve over many CTAs, and a logistic one (grid barriers in its scan)."""
    prec = 10 ** np.random.default_rng(3).uniform(-1, 1, 16)
    a = pmcmc.solve(pmcmc.DensityModel.diag_gaussian(prec),
                    pmcmc.ParallelMALASampler(0.05, T=2000, jacobian="diag", dtype=np.float32),
                    np.zeros(16, np.float32), seed=5, handle=h, return_logp=True)
    rng = np.random.default_rng(4)
    X = rng.standard_normal((300, 40)) / 6
    b = pmcmc.solve(pmcmc.DensityModel.logistic(X, (rng.random(300) < 0.5).astype(float)),
                    pmcmc.ParallelMALASampler(0.02, T=1000, dtype=np.float32),
                    np.zeros(40, np.float32), seed=5, handle=h, return_logp=True)
    assert a[1]["converged"] and b[1]["converged"]
    return a, b


@pytest.mark.parametrize("kind", ["grid_barrier", "mailbox"])
def test_wait_gives_up_at_its_bound_and_handle_stays_usable(kind):
    h = pmcmc.Handle(0)
    r = h.check_wait_bound(kind)
    assert r["status"] == L.ERR_TIMEOUT, r
    assert "reached its bound" in r["message"]
    # bounds: 2^22 polls of the barrier's word, 2e9 SM cycles for the message
    assert 1.0 <= r["wait_ms"] <= 20000.0, r
    for got, want in zip(_solves(h), _solves(pmcmc.Handle(0))):
        assert got[1]["iters"] == want[1]["iters"]
        for i in (0, 2, 3):
            np.testing.assert_array_equal(got[i], want[i])
