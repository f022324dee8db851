"""The column kernels themselves, pinned, in both precisions and on both sides
of the rules that choose them or a one-launch step: against the oracle, with
the launches' names.  Tolerances FP64 1e-12, split 1e-5."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
CASES = [
    (2, 3, [[0, 1], [1, 0], [3, 0]], [2, 64, 64, 64, 1], 257),
    (3, 2, [[1, 0, 0], [0, 2, 0], [0, 0, 2]], [3, 33, 7, 1], 65),
    (1, 1, None, [1, 5, 3, 1], 1),
    (2, 4, [[2, 1]], [2, 20, 36, 1], 31),       # top degree 3 below K
    (2, 7, None, [2, 48, 24, 40, 1], 33),       # 36 slots: the largest taken
    (4, 3, None, [4, 32, 32, 1], 300),
    (3, 2, None, [3, 100, 70, 1], 50),
    (2, 2, None, [2, 20, 64, 1], 1300),         # more threads than fit at once
    (4, 3, None, [4, 16, 64, 1], 600),
]


@pytest.fixture
def pin():
    def set_(fwd, adj):
        api.tune_force(0, fwd)
        api.tune_force(1, adj)
    yield set_
    set_(-1, -1)


def _gradient(net, X):
    g, r = net.grad(), api.SeedRule(api.SEED_HALFSQ)
    api.profile_enable(True)
    api.profile_read()
    loss, T = g.rule_batch(X, r, want_t=True)
    names = api.profile_read()
    api.profile_enable(False)
    out = T, g.read(), loss, names
    r.free(); g.free()
    return out


@pytest.mark.parametrize("d0,k,seeds,dims,npts", CASES)
@pytest.mark.parametrize("prec,tol", [(api.PREC_F64, 1e-12), (api.PREC_SPLIT, 1e-5)])
def test_pinned_column_step(d0, k, seeds, dims, npts, prec, tol, pin):
    w = xavier_weights(dims, 23)
    w[np.arange(len(w)) % 6 == 0] += 0.04
    X = np.random.default_rng(3).uniform(-1, 1, (npts, d0))
    ts, ref = api.TableSet(d0, k, seeds), po.Tables(d0, k, seeds)
    net = api.Net(ts, dims, weights=w, precision=prec)
    pin(4, 4)
    T, gd, loss, names = _gradient(net, X)
    assert "k_point" not in names and {"k_bell_fwd", "k_bell_adj", "k_bell_adj_l2"} <= set(names)
    gref, Tref, lref, _ = po.grad_batch(ref, dims, w, X)
    assert rel_err(T, Tref) < tol and rel_err(gd, gref) < tol
    assert abs(loss - lref) <= tol * abs(lref)
    j = api.SeedRule(api.SEED_JROW, [(1.0, ts.na, 0), (0.5, 1, 1)])
    rows = api.jacobian_rows(net, X, j)[0]
    rref = po.grad_batch(ref, dims, w, X, kind=po.SEED_JROW, terms=[(1.0, ts.na, 0), (0.5, 1, 1)])[3]
    assert rel_err(rows, rref) < tol
    j.free(); net.free(); ts.free()


@pytest.mark.parametrize("prec,row", [(api.PREC_F64, 16), (api.PREC_SPLIT, 32)])
@pytest.mark.parametrize("d0,k,line", [(2, 3, 512), (4, 3, 1024)])
def test_the_rule_takes_them_from_its_line(d0, k, line, prec, row, pin):
    """One row of neurons a point: line points make the rule's bytes.  On both
    sides the step agrees with the oracle; from the line on it has the bits of
    the pinned columns (which differ from the others' in the order of sums)."""
    dims = [d0, row, row, 1]
    ts, ref = api.TableSet(d0, k), po.Tables(d0, k)
    w = xavier_weights(dims, 5)
    net = api.Net(ts, dims, weights=w, precision=prec)
    tol = 1e-12 if prec == api.PREC_F64 else 1e-5
    for npts in (line - 1, line):
        X = np.random.default_rng(npts).uniform(-1, 1, (npts, d0))
        pin(4, 4)
        pinned = net.eval(X)
        pin(-1, 4)                               # the forward by rule, no one-launch step
        T = net.eval(X)
        pin(-1, -1)
        assert rel_err(T, po.grad_batch(ref, dims, w, X)[1]) < tol
        if npts == line:
            assert np.array_equal(T, pinned)
        elif k > 2:
            assert not np.array_equal(T, pinned)
    net.free(); ts.free()
