"""FP32 marginals of trees past 3,072 states, which the general backward kernel takes, through tree
switches: within 1e-5 of the oracle's, as everywhere."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_marginals_through_switches():
    import pyoracle

    from argweaver_gb300 import api
    from argweaver_gb300.sim import simulate

    p = simulate(299, 40, 13, compress=10, ntimes=32, popsize=1e5, missing=0.005)
    assert p.ntrees >= 8 and api.cells(p) > 3072 * p.seqlen
    fw, _ = pyoracle.forward(p)
    want = pyoracle.posterior(p, fw, pyoracle.backward(p))
    assert np.max(np.abs(api.posterior(p, precision="fp32") - want)) <= 1e-5
