"""FP64 columns far below the scale that the chain expects: one tree without recombination and
sites that no state explains together under the infinite-sites penalty, so that whole columns
drop by the penalty (more than 40 powers of two: scaled a second time), and emissions below FP64's
normal numbers (1e-306). The forward table against the oracle at 1e-12 relative per cell, marginals
at 1e-10.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(k, columns, seed, penalty, rho):
    from argweaver_gb300.sim import simulate

    p = simulate(k - 1, columns, seed, compress=10, missing=0.005, rho=max(rho, 1e-14))
    p.rho = 10 * rho
    for i, c in enumerate(range(10, columns, 7)):  # the new haplotype shares a base with one leaf, another each time
        p.seqs[:, c] = ord("A")
        p.seqs[[i % (k - 1), k - 1], c] = ord("C")
    p.infsites_penalty = penalty
    return p


@pytest.mark.parametrize("k,columns,penalty,rho", [(8, 150, 1e-20, 1e-22), (8, 150, 1e-150, 1e-22), (30, 100, 1e-60, 1e-22),
                                                   (8, 150, 1e-306, 1.6e-8), (60, 80, 1e-306, 1.6e-8)])
def test_penalised_columns(k, columns, penalty, rho):
    import pyoracle

    from argweaver_gb300 import api

    p = _problem(k, columns, 40 + k, penalty, rho)
    fw, lnl = pyoracle.forward(p)
    if rho < 1e-16:
        p.infsites_penalty = 1.0
        drop = (pyoracle.forward(p)[1] - lnl) / len(range(10, columns, 7))
        assert drop > 40 * np.log(2)  # of a site, on average
        p.infsites_penalty = penalty
    a = api.run_batch([p], want_posterior=True)[0]
    big = fw > 1e-280
    assert np.max(np.abs(a.forward - fw)[big] / fw[big]) <= 1e-12
    assert abs(a.loglik - lnl) <= 1e-12 * abs(lnl)
    post = pyoracle.posterior(p, fw, pyoracle.backward(p))
    big = post > 1e-200
    assert np.max(np.abs(a.posterior[big] - post[big]) / post[big]) <= 1e-10
