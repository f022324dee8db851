"""The one-thread-per-neuron Bell kernels of small carried sets and the
analytic first-layer adjoint, against the oracle: closures and dense sets up
to the largest the rule takes, widths that are no multiple of a warp or of
four, a single point and point counts around the blocks' edges, the
gradient, the loss, every derivative and the Jacobian rows.

Tolerances are those of the whole step elsewhere: 1e-12 in FP64 and 1e-5 on
the split path."""
import numpy as np
import pytest

import pyoracle as po
from conftest import per_order_error, rel_err, xavier_weights
from dnnf90_b200 import api

CASES = [
    (2, 3, [[0, 1], [1, 0], [3, 0]], [2, 64, 64, 64, 1], 257),
    (3, 2, [[1, 0, 0], [0, 2, 0], [0, 0, 2]], [3, 33, 7, 1], 65),
    (1, 1, None, [1, 5, 3, 1], 1),
    (2, 4, [[2, 1]], [2, 20, 36, 1], 31),       # top degree 3 below K
    (2, 7, None, [2, 48, 24, 40, 1], 33),       # 36 slots: the largest taken
    (4, 3, None, [4, 32, 32, 1], 300),          # 35 slots
    (3, 2, None, [3, 100, 70, 2], 50),
]
BIG = [
    (4, 7, None, [4, 8, 8, 1], 3),              # slots split over blocks
    (4, 7, None, [4, 44, 20, 1], 9),
    (3, 5, None, [3, 70, 12, 1], 130),
    (2, 8, None, [2, 17, 16, 1], 64),
]


def _step(d0, k, seeds, dims, npts, prec):
    rng = np.random.default_rng(3)
    w = xavier_weights(dims, 23)
    w[np.arange(len(w)) % 6 == 0] += 0.04
    X = rng.uniform(-1, 1, (npts, d0))
    ts, ref = api.TableSet(d0, k, seeds), po.Tables(d0, k, seeds)
    net = api.Net(ts, dims, weights=w, precision=prec)
    g = net.grad()
    r = api.SeedRule(api.SEED_HALFSQ)
    loss, T = g.rule_batch(X, r, want_t=True)
    gd = g.read()
    gref, Tref, lref, _ = po.grad_batch(ref, dims, w, X)
    tol = 1e-12 if prec == api.PREC_F64 else 1e-5
    if dims[-1] == 1:
        assert max(per_order_error(T, Tref, ref.deg).values()) < tol
    assert rel_err(gd, gref) < tol, rel_err(gd, gref)
    assert abs(loss - lref) <= tol * abs(lref)
    if dims[-1] == 1:
        terms = [(1.0, ts.na, 0), (0.5, 1, 1)]
        j = api.SeedRule(api.SEED_JROW, terms)
        rows, _, _ = api.jacobian_rows(net, X, j)
        _, _, _, rref = po.grad_batch(ref, dims, w, X, kind=po.SEED_JROW, terms=terms)
        assert rel_err(rows, rref) < tol
        j.free()
    r.free(); g.free(); net.free(); ts.free()


@pytest.mark.gpu
@pytest.mark.parametrize("d0,k,seeds,dims,npts", CASES + BIG)
@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
def test_step_against_the_oracle(d0, k, seeds, dims, npts, prec):
    _step(d0, k, seeds, dims, npts, prec)


@pytest.mark.gpu
def test_small_sets_are_not_timed():
    """The column kernels run by rule: a launch with many waves of work on a
    small set adds no line to the autotuner's report."""
    ts = api.TableSet(2, 3, [[0, 1], [1, 0], [3, 0]])
    dims = [2, 52, 52, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 1))
    g = net.grad()
    r = api.SeedRule(api.SEED_HALFSQ)
    g.rule_batch(np.random.default_rng(0).uniform(-1, 1, (4096, 2)), r)
    assert not [t for t in api.tune_report() if t[3:5] == (5, 52)]
    r.free(); g.free(); net.free(); ts.free()
