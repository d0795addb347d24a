"""A problem's FP64 path, marginals and log-likelihood do not depend on what else is asked for:
its own table, or another problem's."""

import numpy as np
import pytest

from argweaver_gb300 import api, capi
from argweaver_gb300.server import Server
from argweaver_gb300.sim import simulate

pytestmark = pytest.mark.gpu


def _batch(n):
    probs = [simulate(4 + 9 * (i % 4), 250 + 31 * i, 60 + i, missing=0.005) for i in range(n)]
    return probs, [np.random.default_rng(i).random(p.seqlen) for i, p in enumerate(probs)]


@pytest.mark.parametrize("n", [1, 3, 20])
def test_with_and_without_tables(n):
    probs, u = _batch(n)
    a = api.run_batch(probs, want_forward=False, want_path=True, want_posterior=True, uniforms=u)
    b = api.run_batch(probs, want_forward=True, want_path=True, want_posterior=True, uniforms=u)
    for x, y in zip(a, b):
        assert np.array_equal(x.path, y.path) and x.loglik == y.loglik
        assert np.array_equal(x.posterior, y.posterior)


def test_one_table_of_a_batch():
    probs, u = _batch(4)
    want = api.run_batch(probs, want_forward=False, want_path=True, want_posterior=True, uniforms=u)
    tables = api.run_batch(probs)
    bound, outs, got, keep = api._bind_batch(probs, "fp64", False, True, True, u)
    fw = np.empty_like(tables[2].forward)
    outs[2].forward = fw.ctypes.data
    assert capi.load().awg_run_batch(bound, outs, len(probs), capi.AWG_FP64) == 0
    assert np.array_equal(fw, tables[2].forward)
    for (r, _), w in zip(got, want):
        assert np.array_equal(r.path, w.path) and np.array_equal(r.posterior, w.posterior)


def test_resampling_behind_a_wanted_table():
    """The columns that a path is drawn from are the same before and after the table is handed over."""
    p = simulate(20, 1500, seed=21, missing=0.005)
    us = [np.random.default_rng(i).random(p.seqlen) for i in range(4)]
    want = [api.sample_path(p, u) for u in us]
    with Server(device_bytes=1 << 30, max_inflight=1, max_batch=1) as srv:
        t = srv.submit(p, precision="fp64", want_forward=True, uniforms=us[0], resident=True)
        r = srv.wait(t, timeout=120)
        assert np.array_equal(r.path, want[0])
        assert np.array_equal(r.forward, api.forward(p)[0])
        for u, w in zip(us[1:], want[1:]):
            assert np.array_equal(srv.resample(t, u), w)
        srv.release(t)


@pytest.mark.parametrize("n", [2, 18])
def test_marginals_wanted_later_in_a_context(n):
    """A context's first batch wants none (nothing is made for them), a later one does."""
    probs, u = _batch(n)
    want = api.run_batch(probs, precision="fp32", want_forward=False, want_path=True, want_posterior=True, uniforms=u)
    with api.BatchContext() as c:
        for post in (False, True, False, True):
            c.launch(probs, precision="fp32", want_posterior=post, uniforms=u)
            for r, w in zip(c.finish(), want):
                assert np.array_equal(r.path, w.path)
                assert not post or np.array_equal(r.posterior, w.posterior)


def test_paths_longer_than_the_staging():
    """18 problems of a million columns (72 MB of paths, in pieces of 32 MB through two buffers), one
    of them without a path."""
    p = simulate(3, 1000003, 9, ntimes=8, rho=1e-11)
    u = [np.random.default_rng(i).random(p.seqlen) for i in range(18)]
    bound, outs, got, keep = api._bind_batch([p] * 18, "fp32", False, True, False, u)
    outs[4].path = None
    assert capi.load().awg_run_batch(bound, outs, 18, capi.AWG_FP32) == 0
    for q in (0, 3, 5, 7, 8, 9, 16, 17):  # pieces end in problems 8 and 16
        assert np.array_equal(got[q][0].path, api.sample_path(p, u[q], precision="fp32"))
    api.release_memory()
