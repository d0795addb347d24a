"""The FP32 forward kernel on trees of long branches (large N), whose same-branch rows are longer
than the registers hold and too long to stage two trees of: rows by a bulk copy at the tree's
start, or from global memory. Against the oracle's FP64 table, 1e-5 an entry (columns sum to 1),
and its log-likelihood, 1e-6 of its size.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# three, four and eight states a thread, 20, 24 and 32 time points; the last three without rows in
# shared memory
@pytest.mark.parametrize("k,popsize,ntimes", [(50, 1e5, 32), (80, 1e5, 32), (40, 1e6, 32), (130, 1e5, 32), (60, 1e6, 24),
                                              (70, 1e6, 20), (140, 1e5, 20), (50, 1e7, 32), (100, 1e6, 32), (160, 1e7, 20)])
def test_fp32_rows_not_staged(k, popsize, ntimes):
    import pyoracle

    from argweaver_gb300 import api
    from argweaver_gb300.sim import simulate

    p = simulate(k - 1, 60, 100 + k, compress=10, ntimes=ntimes, popsize=popsize, missing=0.005)
    fw, lnl = pyoracle.forward(p)
    a = api.run_batch([p], precision="fp32")[0]
    assert np.max(np.abs(a.forward - fw)) <= 1e-5
    assert abs(a.loglik - lnl) <= 1e-6 * abs(lnl)


@pytest.mark.parametrize("k,popsize,ntimes", [(30, 1e6, 32), (40, 1e7, 32), (50, 1e6, 32), (60, 1e6, 24), (160, 1e5, 32),
                                              (90, 1e7, 20), (160, 1e7, 20)])
def test_fp32_rows_past_the_registers_in_one_tree(k, popsize, ntimes):
    import pyoracle

    from argweaver_gb300 import api
    from argweaver_gb300.sim import simulate

    p = simulate(k - 1, 70, 300 + k, compress=10, ntimes=ntimes, popsize=popsize, missing=0.005, rho=1e-14)
    assert p.ntrees == 1
    fw, lnl = pyoracle.forward(p)
    a = api.run_batch([p], precision="fp32")[0]
    assert np.max(np.abs(a.forward - fw)) <= 1e-5
    assert abs(a.loglik - lnl) <= 1e-6 * abs(lnl)
