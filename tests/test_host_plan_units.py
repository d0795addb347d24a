"""The host's plan of a batch, shared out over threads by units of trees: sizes, the first error of
a batch, and the transposed sequences and column classes at the edges of its 8-byte blocks, 16-byte
vectors and 256-column tiles."""

import dataclasses

import numpy as np
import pytest

from argweaver_gb300 import api, capi
from argweaver_gb300.sim import simulate


def _cells(probs):
    lib = capi.load()
    bound = [api._Bound(p) for p in probs]
    arr = (capi.AwgProblem * len(probs))(*[b.c for b in bound])
    out = np.zeros(len(probs), dtype=np.int64)
    if lib.awg_problems_cells(arr, len(probs), out.ctypes.data) != 0:
        return capi.last_error()
    return list(out)


@pytest.fixture(scope="module")
def many_trees():
    return simulate(30, 20000, 5, compress=10, ntimes=20, rho=4e-7)


def test_cells_of_many_units(many_trees):
    assert many_trees.ntrees > 4000  # several units of trees, several threads
    small = simulate(4, 50, 6, compress=10, ntimes=8)
    assert _cells([small, many_trees, small]) == [p.cells() for p in (small, many_trees, small)]


@pytest.mark.parametrize("what,message", [("age", "node age out of range"), ("parent", "malformed tree"),
                                          ("spr", "SPR nodes out of range"), ("len", "block length < 1")])
def test_first_error_of_a_batch(many_trees, what, message):
    bad = dataclasses.replace(many_trees, ages=many_trees.ages.copy(), ptrees=many_trees.ptrees.copy(),
                              sprs=many_trees.sprs.copy(), blocklens=many_trees.blocklens.copy())
    b = many_trees.ntrees - 2  # in a late unit
    if what == "age":
        bad.ages[b, 3] = 99
    elif what == "parent":
        bad.ptrees[b, 0] = bad.ptrees[b, 1] = bad.ptrees[b, 2]
        bad.ptrees[b, 2] = bad.nnodes
    elif what == "spr":
        bad.sprs[b, 0] = bad.nnodes
    else:
        bad.blocklens[b] = 0
    worse = dataclasses.replace(many_trees, times=many_trees.times[::-1].copy())
    assert message in _cells([many_trees, bad, worse])
    assert _cells([many_trees, bad, worse]).startswith("problem 1:")
    assert _cells([worse, bad]) == "problem 0: times not increasing"


@pytest.mark.gpu
@pytest.mark.parametrize("k,columns", [(3, 15), (7, 16), (8, 17), (9, 255), (15, 256), (16, 257), (17, 300),
                                       (25, 520)])
def test_columns_at_the_edges(k, columns):
    import pyoracle

    p = simulate(k - 1, columns, 80 + k, compress=10, ntimes=20, missing=0.05, rho=1e-7)
    r = api.run_batch([p], precision="fp64")[0]
    fw, ll = pyoracle.forward(p)
    # FP64 sums in another order over a few hundred columns
    assert np.max(np.abs(r.forward - fw)) <= 1e-10 * np.max(np.abs(fw))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_packed_downloads_equal_alone(precision):
    probs = [simulate(k, 100 + 7 * k, 60 + k, compress=10, ntimes=20, missing=0.01) for k in range(3, 9)]
    us = [np.random.default_rng(i).random(p.seqlen) for i, p in enumerate(probs)]
    for p, u, r in zip(probs, us, api.run_batch(probs, precision=precision, want_path=True, uniforms=us)):
        one = api.run_batch([p], precision=precision, want_path=True, uniforms=[u])[0]
        assert np.array_equal(r.path, one.path) and r.loglik == one.loglik
