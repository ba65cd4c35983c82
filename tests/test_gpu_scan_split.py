"""The affine scan's split (chunks of columns, runs inside a chunk, blocks of coordinates,
launches of a long scan) at its edges, against the sequential FP64 recurrence."""
import numpy as np
import pytest

import oracle as O
import pmcmc

pytestmark = pytest.mark.gpu

# |A| <= 0.99: a rounding error of a step decays, so the error stays within about
# eps / (1 - 0.99) of the largest state (itself about 1 / sqrt(1 - 0.99^2) = 7)
TOL = {np.float32: 100 * 1.2e-7 * 10, np.float64: 100 * 2.3e-16 * 10}


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("D,T", [
    (1, 7), (1, 9), (2, 4735), (2, 4737),       # one column past full chunks
    (15, 1000), (255, 300), (256, 300), (257, 300), (513, 121),  # blocks of coordinates
    (100, 37889), (3, 160_001),                 # long chunks; two launches by window
    (600, 14_001),                              # launches by L2 (FP64)
])
def test_scan_split_edges(h, dt, D, T):
    rng = np.random.default_rng(D + T)
    A = rng.uniform(-0.99, 0.99, (D, T)).astype(dt)
    B = rng.standard_normal((D, T)).astype(dt)
    s0 = rng.standard_normal(D).astype(dt)
    R = O.scan_seq(A.astype(np.float64), B.astype(np.float64), s0.astype(np.float64))
    np.testing.assert_allclose(pmcmc.solve_affine_scan_diag(A, B, s0, handle=h), R, rtol=0,
                               atol=TOL[dt])


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_scan_keeps_zero_states_and_carries_nonfinite_ones(h, dt):
    D, T = 4, 40_000
    A = np.full((D, T), 1.01, dt)   # composed over all columns this overflows
    B = np.zeros((D, T), dt)
    s0 = np.zeros(D, dt)
    A[1], s0[1] = 0.5, 1.0
    B[1, 20_000] = np.nan           # from there on, and in no other coordinate
    A[2] = 1.0
    B[2, 5] = np.inf
    A[2, 30_000] = 0.0              # inf * 0
    S = pmcmc.solve_affine_scan_diag(A, B, s0, handle=h)
    assert np.all(S[0] == 0) and np.all(S[3] == 0)
    assert np.isfinite(S[1, :20_000]).all() and np.isnan(S[1, 20_000:]).all()
    assert np.all(S[2, 5:30_000] == np.inf) and np.isnan(S[2, 30_000:]).all()
