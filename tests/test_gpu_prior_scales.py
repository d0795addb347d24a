"""A given first column on any scale that FP64 holds: the path does not see the scale (the columns
are scaled by powers of two as they go)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,columns,seed,first", [(6, 400, 5, None), (40, 200, 6, None), (10, 300, 0, 1)])
def test_prior_scales(k, columns, seed, first):
    from argweaver_gb300 import api
    from argweaver_gb300.sim import simulate

    rho = 1.6e-8
    if first:  # a first tree of one column: the prior goes straight through a switch
        rho = 4e-7
        seed = next(s for s in range(100) if simulate(k, columns, s, rho=rho, missing=0.005).blocklens[0] == first)
    p = simulate(k, columns, seed, rho=rho, missing=0.005)
    u = np.random.default_rng(seed).random(p.seqlen)
    top = np.where(p.ptrees[0] >= 0, p.ages[0][np.maximum(p.ptrees[0], 0)], p.ntimes - 2)
    S = int(np.maximum(top - p.ages[0] + 1, 0).sum())
    spread = np.exp2(-np.random.default_rng(1).integers(1, 6, S).astype(float))
    spread /= 2.0 ** np.ceil(np.log2(spread.sum()))  # sums to between 1/2 and 1
    one = np.where(np.arange(S) == S // 3, 0.75, 0.0)
    for prior in (spread, one):
        want = api.sample_path_conditioned(p, prior=prior, uniforms=u)
        # FP64's largest exponents (2^1023 and more in one time bin among them) and small normal numbers
        for e in (300, 900, 1000, 1022, 1024, -600, -1000):
            scaled = np.ldexp(prior, e)
            assert np.isfinite(scaled.sum())
            assert np.array_equal(api.sample_path_conditioned(p, prior=scaled, uniforms=u), want), e
