"""The warp's walk over the recombination draws (awg_sample_recombinations) against the oracle:
trees of more than 32 nodes (a state found over several node groups), more candidates than
lanes (32 time points), runs of more than 32 columns between events, one-column trees, external
and internal. Bar: the same columns, nodes, times and number of draws."""

import numpy as np
import pytest

from test_recomb_sampler import stress_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,L,T,internal,rho,seed", [
    (3, 500, 20, False, 1.6e-8, 1), (40, 3000, 32, False, 1.6e-8, 2), (80, 2500, 20, False, 3e-8, 3),
    (20, 1500, 16, False, 4e-7, 4), (33, 2500, 32, True, 1.6e-8, 5)])
def test_walk_matches_oracle(k, L, T, internal, rho, seed):
    import pyoracle

    from argweaver_gb300 import api
    from argweaver_gb300.sim import leaf_cut, simulate

    p = simulate(k, L, seed, ntimes=T, rho=rho)
    if internal:
        p = leaf_cut(p)
    fw, _ = pyoracle.forward(p)
    path = pyoracle.traceback(p, fw, pyoracle.rand_uniforms(seed, p.seqlen))
    for q in (path, stress_path(p, path, seed)):
        u = np.random.default_rng(seed).random(2 * p.seqlen + 2)
        o = pyoracle.sample_recombinations(p, q, u)
        pos, node, time, used = api.sample_recombinations(p, q, u)
        np.testing.assert_array_equal(pos, o[0])
        np.testing.assert_array_equal(node, o[1])
        np.testing.assert_array_equal(time, o[2])
        assert used == o[3]
