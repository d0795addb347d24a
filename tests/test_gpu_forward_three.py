"""The FP32 forward kernel with three states an owner thread (769 to 1152 states), rows staged
and not, 21 time points or more, against the FP64 forward table of the same problem.

Tolerance: the FP32 path's bar is 1e-5 relative to FP64; columns sum to 1, so the table's 2-norm
differs by at most that share, and the log-likelihood by 1e-6 of its size.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,ntimes,kw", [(140, 20, {}), (190, 20, {}), (115, 32, {}),
                                         (40, 32, dict(popsize=3e5))])
def test_three_states_a_thread(k, ntimes, kw):
    from argweaver_gb300 import api
    from argweaver_gb300.sim import simulate

    p = simulate(k - 1, 250, 4000 + k, compress=10, ntimes=ntimes, missing=0.005, **kw)
    assert 768 < p.nstates_per_tree().max() <= 1152
    a = api.run_batch([p], precision="fp32")[0]
    b = api.run_batch([p], precision="fp64")[0]
    assert np.linalg.norm(a.forward - b.forward) <= 1e-5 * np.linalg.norm(b.forward)
    assert abs(a.loglik - b.loglik) <= 1e-6 * abs(b.loglik)
