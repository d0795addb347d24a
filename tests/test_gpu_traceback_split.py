"""The FP32 path's decomposed draw: chunks and trees of every length, tables staged in three
buffers, in two, or not at all, external and cut trees, against the oracle's decomposed draw given
the GPU's own next state and forward table.

Tolerance: the oracle computes in FP64, so a draw may differ only where the uniform falls within
FP32 rounding (some 1e-6) of a boundary: at most one in these few thousand columns.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (a tree's columns come in chunks of 32)
CASES = [dict(k=3, columns=700, ntimes=4), dict(k=20, columns=1500, ntimes=20, rho=3e-7),
         dict(k=20, columns=33, ntimes=20, rho=1e-12), dict(k=20, columns=2050, ntimes=20, rho=1e-12),
         dict(k=64, columns=400, ntimes=20), dict(k=140, columns=250, ntimes=32),
         dict(k=40, columns=600, ntimes=32, popsize=3e5),
         dict(k=30, columns=2000, ntimes=20, internal=True, missing=0.02)]


def _problem(k, columns, ntimes, seed, internal=False, missing=0.005, **kw):
    from argweaver_gb300 import refapi
    from argweaver_gb300.sim import simulate

    p = simulate(k if internal else k - 1, columns, seed, compress=10, ntimes=ntimes,
                 missing=missing, add_thread=not internal, **kw)
    if internal:
        refapi.srand(seed)
        path, _ = refapi.sample_arg_removal_path_uniform(p)
        p = refapi.as_problem(p, refapi.remove_arg_thread_path(p, path), internal=True)
    return p


@pytest.mark.parametrize("case", range(len(CASES)))
def test_split_draw_forms(case):
    from argweaver_gb300 import api
    import pyoracle

    p = _problem(seed=7300 + case, **CASES[case])
    # uniforms spread over all scales, so that draws leave a state more often than one in a thousand
    rng = np.random.default_rng(case)
    u = rng.random(p.seqlen)
    u[::7] = 1.0 - 10.0 ** rng.uniform(-4, 0, u[::7].shape)
    r = api.run_batch([p], precision="fp32", want_path=True, uniforms=[u])[0]
    ref = pyoracle.traceback_split(p, r.forward.astype(np.float64), u, given=r.path)
    assert np.count_nonzero(ref != r.path) <= 1
    alone = api.run_batch([p] * 3, precision="fp32", want_forward=False, want_path=True, uniforms=[u] * 3)
    assert all(np.array_equal(x.path, r.path) for x in alone)
