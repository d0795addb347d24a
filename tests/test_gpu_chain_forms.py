"""The FP64 forward and the backward chain kernel's forms (two lanes a state, states per owner
thread) against the oracle, at the repository's bars: the FP64 forward table 1e-12 relative per
cell, FP64 posterior marginals 1e-10 relative, FP32 marginals 1e-5 of FP64.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# states below and above 192, 384, 768 and 1536 (the forms' limits), the smallest trees, and
# 16, 20 and 32 time points (the bins' split over the reduction warps)
SHAPES = [(3, 300, 20), (6, 300, 16), (10, 300, 32), (20, 250, 20), (24, 250, 16), (40, 200, 20),
          (52, 200, 20), (30, 150, 32), (110, 120, 20), (130, 120, 20), (205, 60, 32), (216, 60, 32)]


def _problem(k, columns, ntimes, seed, **kw):
    from argweaver_gb300.sim import simulate

    return simulate(k - 1, columns, seed, compress=10, ntimes=ntimes, missing=0.005, **kw)


def _check(p):
    import pyoracle

    from argweaver_gb300 import api

    a = api.run_batch([p], want_posterior=True)[0]
    fw, lnl = pyoracle.forward(p)
    assert np.max(np.abs(a.forward - fw) / np.maximum(fw, 1e-300)) <= 1e-12
    assert abs(a.loglik - lnl) <= 1e-12 * abs(lnl)
    post = pyoracle.posterior(p, fw, pyoracle.backward(p))
    big = post > 1e-200
    assert np.max(np.abs(a.posterior[big] - post[big]) / post[big]) <= 1e-10
    f = api.run_batch([p], precision="fp32", want_forward=False, want_posterior=True)[0]
    assert np.max(np.abs(f.posterior - post)) <= 1e-5


@pytest.mark.parametrize("k,columns,ntimes", SHAPES)
def test_chain_forms(k, columns, ntimes):
    _check(_problem(k, columns, ntimes, 5000 + k))


@pytest.mark.parametrize("rho,columns", [(4e-7, 500), (1e-11, 1500)])
def test_chain_short_and_long_trees(rho, columns):
    """Trees of one to a few columns (a column is scaled at every switch), and one tree over many
    windows of column classes."""
    _check(_problem(12, columns, 20, 78, rho=rho))


def test_chain_mixed_sizes_equal_alone():
    """Instances of different forms in one launch give what they give alone."""
    from argweaver_gb300 import api

    probs = [_problem(k, 150, 20, 700 + k) for k in (3, 30, 70, 130, 18)]
    for p, r in zip(probs, api.run_batch(probs, want_posterior=True)):
        one = api.run_batch([p], want_posterior=True)[0]
        assert np.array_equal(r.forward, one.forward) and r.loglik == one.loglik
        assert np.array_equal(r.posterior, one.posterior)


@pytest.mark.parametrize("k,columns", [(12, 300), (60, 200), (110, 120)])
def test_fp32_marginals_through_one_column_trees(k, columns):
    """Trees of one column end where they begin: their low parts replace the later tree's only once
    every owner has read those. The same marginals on every run, within 1e-5 of FP64's."""
    from argweaver_gb300 import api

    p = _problem(k, columns, 20, 31 + k, rho=2e-6)
    assert np.mean(p.blocklens == 1) > 0.5
    want = api.posterior(p)
    runs = [api.posterior(p, precision="fp32") for _ in range(5)]
    assert np.max(np.abs(runs[0] - want)) <= 1e-5
    assert all(np.array_equal(r, runs[0]) for r in runs[1:])
