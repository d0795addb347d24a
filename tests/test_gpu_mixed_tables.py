"""Batches in which one problem's tables do not fit shared memory: the small problems beside it
give what they give alone, bit for bit, and the oracle's values (the FP64 forward table 1e-12
relative per cell, FP64 marginals 1e-10).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(k, columns, seed, popsize=1e5, ntimes=32):
    from argweaver_gb300.sim import simulate

    return simulate(k - 1, columns, seed, compress=10, ntimes=ntimes, popsize=popsize, missing=0.005)


def _sizes(p):
    """The largest tree's states, and the largest tree's same-branch row entries."""
    top = np.where(p.ptrees >= 0, np.take_along_axis(p.ages, np.maximum(p.ptrees, 0), 1), p.ntimes - 2)
    m = np.maximum(top - p.ages + 1, 0).astype(np.int64)
    return int(m.sum(1).max()), int((m * m).sum(1).max())


def test_fp64_small_problems_beside_rows_in_global_memory():
    import pyoracle

    from argweaver_gb300 import api

    # two lanes a state up to 192 states, one above
    probs = [_problem(80, 60, 11)] + [_problem(k, 120, 20 + k) for k in (3, 8, 14)]
    S, M = _sizes(probs[0])
    assert S <= 3072 and 40 * S + 8 * M > 200 * 1024  # columns, slots and rows in FP64
    assert any(_sizes(p)[0] <= 192 for p in probs) and any(192 < _sizes(p)[0] <= 384 for p in probs)
    u = [np.random.default_rng(3).random(p.seqlen) for p in probs]
    batch = api.run_batch(probs, want_path=True, want_posterior=True, uniforms=u)
    for p, up, r in zip(probs, u, batch):
        one = api.run_batch([p], want_path=True, want_posterior=True, uniforms=[up])[0]
        assert np.array_equal(r.forward, one.forward) and r.loglik == one.loglik
        assert np.array_equal(r.posterior, one.posterior) and np.array_equal(r.path, one.path)
        fw, lnl = pyoracle.forward(p)
        assert np.max(np.abs(r.forward - fw) / np.maximum(fw, 1e-300)) <= 1e-12
        assert abs(r.loglik - lnl) <= 1e-12 * abs(lnl)
        post = pyoracle.posterior(p, fw, pyoracle.backward(p))
        big = post > 1e-200
        assert np.max(np.abs(r.posterior[big] - post[big]) / post[big]) <= 1e-10


@pytest.mark.parametrize("ntimes,k,popsize,rows,small", [(32, 57, 1e7, 42000, (4, 14, 16)), (20, 90, 1e8, 30000, (3, 57, 76))])
def test_fp32_small_problems_beside_rows_too_long_to_stage(ntimes, k, popsize, rows, small):
    """FP32 tables within 1e-5 of FP64's, an entry each."""
    from argweaver_gb300 import api

    probs = [_problem(k, 40, 5, popsize, ntimes)] + [_problem(x, 100, 30 + x, ntimes=ntimes) for x in small]
    S, M = _sizes(probs[0])
    assert 1536 < S <= 1850 and M > rows  # no form stages these rows twice in 222 KB
    batch = api.run_batch(probs, precision="fp32")
    for p, r, w in zip(probs, batch, api.run_batch(probs)):
        one = api.run_batch([p], precision="fp32")[0]
        assert np.array_equal(r.forward, one.forward) and r.loglik == one.loglik
        assert np.max(np.abs(r.forward - w.forward)) <= 1e-5
        assert abs(r.loglik - w.loglik) <= 1e-6 * abs(w.loglik)


def test_fp32_marginals_beside_rows_in_global_memory():
    from argweaver_gb300 import api

    probs = [_problem(57, 40, 5, 1e7)] + [_problem(x, 100, 30 + x) for x in (4, 14, 16)]
    S, M = _sizes(probs[0])
    assert 4 * M > 190 * 1024  # beside columns and slots, past the 200 KB of a launch
    for p, r in zip(probs, api.run_batch(probs, precision="fp32", want_forward=False, want_posterior=True)):
        assert np.array_equal(r.posterior, api.posterior(p, precision="fp32"))
        assert np.max(np.abs(r.posterior - api.posterior(p))) <= 1e-5
