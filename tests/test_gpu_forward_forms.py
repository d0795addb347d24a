"""The FP32 forward kernel's forms (states per owner thread, rows past the registers, tables
staged or not, the wide CTA) against the FP64 forward table of the same problem.

Tolerance: the FP32 path's bar is 1e-5 relative to FP64; columns sum to 1, so the table's
2-norm differs by at most that share, and the log-likelihood by 1e-6 of its size.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(k, columns, ntimes, seed, **kw):
    from argweaver_gb300.sim import simulate

    return simulate(k - 1, columns, seed, compress=10, ntimes=ntimes, missing=0.005, **kw)


# haplotypes and time points on both sides of each form's limit: 32, 384, 768 and 1536
# states (the FP64 emission kernel stops short of 2000), 21 time points
SHAPES = [(3, 400, 20), (5, 400, 16), (12, 400, 32), (40, 300, 20), (52, 300, 20), (30, 200, 32),
          (100, 250, 20), (120, 250, 20), (64, 200, 32), (190, 150, 32), (205, 150, 32),
          (216, 100, 32)]


@pytest.mark.parametrize("k,columns,ntimes", SHAPES)
def test_fp32_forward_forms(k, columns, ntimes):
    from argweaver_gb300 import api

    p = _problem(k, columns, ntimes, 4000 + k)
    a = api.run_batch([p], precision="fp32")[0]
    b = api.run_batch([p], precision="fp64")[0]
    rel = np.linalg.norm(a.forward - b.forward) / np.linalg.norm(b.forward)
    assert rel <= 1e-5, rel
    assert abs(a.loglik - b.loglik) <= 1e-6 * abs(b.loglik)


@pytest.mark.parametrize("rho,columns", [(4e-7, 700), (1e-11, 2500)])
def test_fp32_forward_short_and_long_trees(rho, columns):
    """Trees of one to a few columns (rows fetched ahead end with the tree), and one tree over
    many windows of column classes."""
    from argweaver_gb300 import api

    p = _problem(20, columns, 20, 77, rho=rho)
    assert (p.blocklens.min() <= 2) if rho > 1e-8 else (p.ntrees == 1)
    a = api.run_batch([p], precision="fp32")[0]
    b = api.run_batch([p], precision="fp64")[0]
    assert np.linalg.norm(a.forward - b.forward) <= 1e-5 * np.linalg.norm(b.forward)
    assert abs(a.loglik - b.loglik) <= 1e-6 * abs(b.loglik)


def test_fp32_forward_mixed_sizes_equal_alone():
    """Instances of different forms in one launch give the tables that they give alone."""
    from argweaver_gb300 import api

    probs = [_problem(k, 200, 20, 900 + k) for k in (3, 40, 70, 130, 8)]
    for p, r in zip(probs, api.run_batch(probs, precision="fp32")):
        one = api.run_batch([p], precision="fp32")[0]
        assert np.array_equal(r.forward, one.forward) and r.loglik == one.loglik
