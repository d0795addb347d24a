"""The FP64 traceback's lots and rounds against the oracle's scan: the same path given the same
uniforms. Half of the uniforms are drawn near 0 and 1, so that draws leave their state at every
place of a round and of a lot (the copied columns of one tree); some are exactly 0, where the
scan's first state is drawn whatever its weight. Sizes: 64 columns a lot and fewer, one
column at a time, trees shorter and longer than a lot, internal-branch trees."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniforms(n, seed):
    rng = np.random.default_rng(seed)
    u = rng.random(n)
    edge = rng.random(n) < 0.5
    u[edge] = np.where(rng.random(n) < 0.5, u * 0.02, 1 - u * 0.02)[edge]
    u[rng.random(n) < 0.002] = 0.0
    return u


@pytest.mark.parametrize("k,L,T,rho,internal", [
    (3, 700, 20, 1.6e-8, False), (9, 2500, 20, 1.6e-8, False), (9, 1500, 20, 1e-11, False),
    (14, 800, 16, 3e-7, False), (33, 900, 20, 1.6e-8, False), (64, 500, 20, 1.6e-8, False),
    (150, 150, 20, 1.6e-8, False), (205, 60, 32, 1.6e-8, False), (12, 900, 20, 1.6e-8, True)])
def test_fp64_traceback_lots(k, L, T, rho, internal):
    import pyoracle

    from argweaver_gb300 import api
    from argweaver_gb300.sim import leaf_cut, simulate

    p = simulate(k - 1, L, 60 + k, ntimes=T, rho=rho, missing=0.005)
    if internal:
        p = leaf_cut(p)
    fw, _ = pyoracle.forward(p)
    for seed in range(3):
        u = _uniforms(p.seqlen, seed)
        r = api.run_batch([p], want_forward=False, want_path=True, uniforms=[u])[0]
        np.testing.assert_array_equal(r.path, pyoracle.traceback(p, fw, u))
