"""Variant columns in FP64 and, on the FP32 path, in double-float, at the edges of the groups that a warp carries
through a tree at once, against the FP64 path's forward table of the same problem.

Tolerance: the FP32 path's bar is 1e-5 relative to FP64 (columns sum to 1, so the table's 2-norm
differs by at most that share), and the log-likelihood by 1e-6 of its size.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(k, columns, ntimes, seed, internal=False, penalty=0.0, missing=0.005, **kw):
    from argweaver_gb300 import refapi
    from argweaver_gb300.sim import simulate

    p = simulate(k if internal else k - 1, columns, seed, compress=10, ntimes=ntimes,
                 missing=missing, add_thread=not internal, **kw)
    if internal:
        refapi.srand(seed)
        path, _ = refapi.sample_arg_removal_path_uniform(p)
        p = refapi.as_problem(p, refapi.remove_arg_thread_path(p, path), internal=True)
    p.infsites_penalty = penalty
    return p


# two leaves; the fewest time points that the simulator takes; one tree over more than a window of columns, with many, few
# and no columns that vary through missing calls alone; most calls missing; trees that leave an
# SM one CTA, and one of fewer warps; cut subtrees; penalised columns
CASES = [dict(k=3, columns=300, ntimes=20), dict(k=4, columns=300, ntimes=4),
         dict(k=20, columns=2100, ntimes=20, rho=1e-11), dict(k=12, columns=1025, ntimes=16, rho=1e-11, missing=0.0),
         dict(k=9, columns=400, ntimes=20, missing=0.7), dict(k=33, columns=500, ntimes=32, rho=3e-7),
         dict(k=150, columns=120, ntimes=32), dict(k=216, columns=100, ntimes=32),
         dict(k=30, columns=500, ntimes=20, internal=True), dict(k=20, columns=500, ntimes=20, penalty=1e-3),
         dict(k=16, columns=500, ntimes=20, penalty=1e-2, internal=True)]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_variant_columns_in_groups(case):
    from argweaver_gb300 import api

    p = _problem(seed=6100 + case, **CASES[case])
    a = api.run_batch([p], precision="fp32")[0]
    b = api.run_batch([p], precision="fp64")[0]
    assert np.linalg.norm(a.forward - b.forward) <= 1e-5 * np.linalg.norm(b.forward)
    assert abs(a.loglik - b.loglik) <= 1e-6 * abs(b.loglik)


def test_persistent_queue_equals_one_cta_a_tree():
    """Trees taken in units from the queue (several instances a CTA) give what they give alone."""
    from argweaver_gb300 import api

    probs = [_problem(k, 250, 20, 40 + k) for k in range(4, 38, 2)]
    for p, r in zip(probs, api.run_batch(probs, precision="fp32")):
        one = api.run_batch([p], precision="fp32")[0]
        assert np.array_equal(r.forward, one.forward) and r.loglik == one.loglik


@pytest.mark.parametrize("case", [0, 2, 3, 4, 5, 8, 9, 10])
def test_fp64_columns_in_groups(case):
    """Against the oracle: FP64 sums in another order over some thousand columns."""
    import pyoracle

    from argweaver_gb300 import api

    p = _problem(seed=6100 + case, **CASES[case])
    fw, _ = pyoracle.forward(p)
    r = api.run_batch([p], precision="fp64")[0]
    assert np.max(np.abs(r.forward - fw)) <= 1e-10 * np.max(np.abs(fw))
