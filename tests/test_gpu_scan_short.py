"""Scans of one chunk of columns (no grid barrier) and of the first few, against the sequential
FP64 recurrence; and with s0 a column of the output's own buffer."""
import numpy as np
import pytest
import torch

import oracle as O
import pmcmc
from pmcmc import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    return pmcmc.Handle(0)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("T", [1, 2, 8, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("D", [1, 5, 100, 256, 257, 700])
def test_short_scans(h, dt, D, T):
    rng = np.random.default_rng(100 * D + T)
    A = rng.uniform(-0.99, 0.99, (D, T)).astype(dt)
    B = rng.standard_normal((D, T)).astype(dt)
    s0 = rng.standard_normal(D).astype(dt)
    R = O.scan_seq(A.astype(np.float64), B.astype(np.float64), s0.astype(np.float64))
    # |A| <= 0.99: rounding errors decay, at most eps / (1 - 0.99) of states of about 7
    np.testing.assert_allclose(pmcmc.solve_affine_scan_diag(A, B, s0, handle=h), R, rtol=0,
                               atol=1000 * np.finfo(dt).eps)


@pytest.mark.parametrize("D,T", [(20, 32), (256, 32), (20, 640)])
def test_entering_state_in_the_output_buffer(h, D, T):
    g = torch.Generator(device="cuda").manual_seed(D + T)
    A = torch.rand((T, D), generator=g, device="cuda") * 0.9
    B = torch.randn((T, D), generator=g, device="cuda")
    S = torch.randn((T, D), generator=g, device="cuda")
    want = pmcmc.solve_affine_scan_diag(A.T, B.T, S[0].clone(), handle=h)
    torch.cuda.synchronize()
    # (T, D) row by row is the (D, T) layout of the C interface; s0 = S[:, 0]
    rc = L.load().pmcmc_affine_scan_diag(h.ptr, 0, D, T, A.data_ptr(), B.data_ptr(), S.data_ptr(),
                                         S.data_ptr(), L.MEM_DEVICE)
    assert rc == L.OK
    assert torch.equal(S.T, want)
