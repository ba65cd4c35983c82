"""pmcmc_autotune times the shape that an untuned solve takes beside its candidates, so that tuning
makes no solve slower."""
import time

import numpy as np
import pytest

import pmcmc
from pmcmc import configs

pytestmark = pytest.mark.gpu


def _best(f, n=30):
    f()
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t)


def _check(model, sampler, x0, N):
    h = pmcmc.Handle(0)
    run = lambda: pmcmc.sample(model, sampler, N, seed=0, initial_params=x0, handle=h)
    before = _best(run)
    r = pmcmc.autotune(model, sampler, x0, seed=0, handle=h)
    assert r["ms"] > 0
    # (a grid of one CTA a column is 1.7 times slower for the small block)
    assert _best(run) <= 1.2 * before


def test_small_block_stays_in_one_cta():
    model, sampler, x0, _ = configs.quickstart_2d()
    _check(model, sampler, x0, 40 * sampler.T)


@pytest.mark.parametrize("T", [1024, 8192])
def test_full_chunk_count_of_the_cost_model(T):
    model, sampler, x0, _ = configs.correlated_gauss_d64(T=T)
    _check(model, sampler, np.asarray(x0), T)
