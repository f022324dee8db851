"""The one-launch step of small networks (point.cu), against the oracle and
against the layer-by-layer kernels, which a pinned variant brings back:
widths about the 8 x 8 tiles and the padded strides, one to three hidden
layers, sets from K = 1 to the largest, closures, several outputs, more points
than blocks, every seed rule and activation.

Both compute the same sums in FP64 in another order, so they agree to
rounding: 1e-12 of each array's largest value, as in the step's other tests."""
import numpy as np
import pytest

import pyoracle as po
from conftest import per_order_error, rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu

CASES = [
    (4, 7, None, [4, 8, 8, 1], 1),
    (4, 7, None, [4, 8, 8, 1], 301),
    (4, 3, None, [4, 32, 32, 1], 7),
    (3, 2, [[1, 0, 0], [0, 2, 0], [0, 0, 2]], [3, 33, 17, 1], 12),
    (2, 3, [[0, 1], [1, 0], [3, 0]], [2, 16, 20, 9, 1], 5),
    (1, 1, None, [1, 1, 1], 3),
    (2, 1, None, [2, 5, 3, 1], 33),
    (3, 4, None, [3, 12, 1], 4),
    (2, 8, None, [2, 7, 24, 1], 2),
    (2, 4, [[2, 1]], [2, 40, 31, 1], 600),
    (8, 2, None, [8, 10, 4, 1], 9),
]


@pytest.fixture
def layered():
    yield lambda on: api.tune_force(0, 0 if on else -1)
    api.tune_force(0, -1)


def _setup(d0, k, seeds, dims, npts, act=0):
    rng = np.random.default_rng(3)
    w = xavier_weights(dims, 23)
    w[np.arange(len(w)) % 6 == 0] += 0.04
    ts = api.TableSet(d0, k, seeds, act)
    return ts, api.Net(ts, dims, weights=w), w, rng.uniform(-1, 1, (npts, d0))


@pytest.mark.parametrize("d0,k,seeds,dims,npts", CASES)
def test_step_against_the_oracle(d0, k, seeds, dims, npts):
    ts, net, w, X = _setup(d0, k, seeds, dims, npts)
    ref = po.Tables(d0, k, seeds)
    g, r = net.grad(), api.SeedRule(api.SEED_HALFSQ)
    n0 = api.launch_count()
    loss, T = g.rule_batch(X, r, want_t=True)
    assert api.launch_count() - n0 <= 2
    gref, Tref, lref, _ = po.grad_batch(ref, dims, w, X)
    assert max(per_order_error(T, Tref, ref.deg).values()) < 1e-12
    assert rel_err(g.read(), gref) < 1e-12
    assert abs(loss - lref) <= 1e-12 * abs(lref)
    terms = [(1.0, ts.na, 0), (0.5, 1, 1)]
    j = api.SeedRule(api.SEED_JROW, terms)
    rows, _, _ = api.jacobian_rows(net, X, j)
    _, _, _, rref = po.grad_batch(ref, dims, w, X, kind=po.SEED_JROW, terms=terms)
    assert rel_err(rows, rref) < 1e-12
    assert max(per_order_error(net.eval(X), Tref, ref.deg).values()) < 1e-12
    for h in (j, r, g, net, ts):
        h.free()


@pytest.mark.parametrize("act", range(5))
def test_step_against_the_layers(layered, act):
    d0, k, dims, npts = 2, 5, [2, 11, 6, 2], 10
    ts, net, w, X = _setup(d0, k, None, dims, npts, act)
    rng = np.random.default_rng(8)
    given = rng.normal(size=(npts, 2, ts.na))
    src = rng.normal(size=(npts, 2))
    rules = [api.SeedRule(api.SEED_HALFSQ),
             api.SeedRule(api.SEED_PINN, [(1.5, 4, 0), (6.0, 2, 1)], 0.3),
             api.SeedRule.system(2, [(1, 1.0, [(1, 2)]), (1, -2.0, [(2, 3), (1, 1)]),
                                     (2, 0.5, [(2, 5)])], wres=[1.0, 3.0], fac=0.7)]
    got = []
    for on in (False, True):
        layered(on)
        out = [net.eval_multi(X)]
        for r in rules:
            g = net.grad()
            if r.kind == api.SEED_SYS:
                loss, t = g.sys_batch(X, r, src, want_t=True)
                out.append(t)
            else:
                loss = g.rule_batch(X, r)
            out += [np.array([loss]), g.read()]
            g.free()
        g = net.grad()
        g.batch(X, given)
        out.append(g.read())
        g.free()
        got.append(out)
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
    for h in (*rules, net, ts):
        h.free()
