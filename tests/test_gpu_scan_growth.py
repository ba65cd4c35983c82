"""The affine scan where its maps leave the range of the type: a state that grows past the
largest number is infinite from there on, as the recurrence leaves it, whatever the split."""
import numpy as np
import pytest

import pmcmc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("D,T", [(3, 2000), (3, 70_000), (100, 65_536), (257, 30_000)])
def test_growing_states_end_infinite(h, dt, D, T):
    # 200^17 and 200^134 are past the range of FP32 and FP64, 200^16 and 200^133 well inside
    A = np.full((D, T), 200.0, dt)
    S = pmcmc.solve_affine_scan_diag(A, np.ones((D, T), dt), np.ones(D, dt), handle=h)
    n = 16 if dt == np.float32 else 133
    R = np.cumsum(np.power(200.0, np.arange(n + 1)))[1:]  # 200^t + ... + 1, from s0 = 1
    # every operation adds positive terms: at most 2 n roundings on the way
    np.testing.assert_allclose(S[:, :n], np.tile(R, (D, 1)), rtol=2 * n * np.finfo(dt).eps)
    assert np.all(S[:, n:] == np.inf)
