"""Forward tables cell by cell, at the sizes where the emission and chain kernels change form: FP64
1e-12 relative to the oracle's, FP32 1e-5 absolute (a column sums to 1)."""

import numpy as np
import pytest

from test_gpu_emissions_df import CASES, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", range(len(CASES)))
def test_cells(case):
    import pyoracle

    from argweaver_gb300 import api

    p = _problem(seed=6100 + case, **CASES[case])
    fw, lnl = pyoracle.forward(p)
    a = api.run_batch([p])[0]
    big = fw > 1e-290
    assert np.max(np.abs(a.forward - fw)[big] / fw[big]) <= 1e-12
    assert abs(a.loglik - lnl) <= 1e-12 * abs(lnl)
    b = api.run_batch([p], precision="fp32")[0]
    assert np.max(np.abs(b.forward - fw)) <= 1e-5
