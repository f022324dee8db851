"""Infinite and NaN seeds: an output takes part in a non-finite value exactly
where its own sum holds it, whatever a kernel pads its tiles with.  Infinities
(and their signs) and NaN are compared entry by entry between the kernels, or
with the formula."""
import numpy as np
import pytest

from conftest import xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture
def pin():
    def set_(fwd, adj):
        api.tune_force(0, fwd)
        api.tune_force(1, adj)
    yield set_
    set_(-1, -1)


def _gradient(net, X, seeds):
    g = net.grad()
    g.batch(X, seeds)
    out = g.read()
    g.free()
    return out


def _same(a, b):
    """Equal classes (finite, NaN, the infinity) of every entry."""
    return (np.array_equal(np.isnan(a), np.isnan(b)) and
            np.array_equal(np.where(np.isinf(a), a, 0.0), np.where(np.isinf(b), b, 0.0)))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("d0,k", [(3, 4), (3, 7), (4, 3), (2, 5)])
def test_tiled_adjoint(d0, k, value, pin):
    """FP64 tiles against the grouped correlation: Sb_0 of the last hidden layer
    (its bias gradient), an infinite seed at each slot in turn."""
    ts, dims = api.TableSet(d0, k), [d0, 32, 32, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 3))
    X = np.random.default_rng(1).uniform(-1, 1, (3, d0))
    lo = 32 * (d0 + 1)
    bias = lo + 33 * np.arange(32)
    for a in range(net.na):
        seeds = np.random.default_rng(a).normal(size=(3, net.na))
        seeds[1, a] = value
        pin(2, 3)
        tiled = _gradient(net, X, seeds)[bias]
        pin(2, 2)
        assert _same(tiled, _gradient(net, X, seeds)[bias]), a
    net.free(); ts.free()


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
@pytest.mark.parametrize("d0,k,n,npts,at", [
    (2, 4, 33, 5000, 4999), (4, 3, 32, 999, 7), (4, 4, 20, 301, 300), (1, 8, 40, 64, 3)])
def test_first_layer_gradient(d0, k, n, npts, at, prec, pin):
    """One hidden layer: with Tb^a infinite at one point, Sb^0 = Tb^a h^a + ...
    and Sb^{e_i} = a_i Tb^a h^{a - e_i} + ..., which Tb^a enters for a_i > 0
    only; dW_i = Sb^0 x_i + Sb^{e_i}."""
    ts, dims = api.TableSet(d0, k), [d0, n, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 4), precision=prec)
    rng = np.random.default_rng(2)
    X = rng.uniform(0.25, 1.0, (npts, d0))
    pin(2, 2)                                   # no one-launch step
    for a in range(0, net.na, max(1, net.na // 9)):
        seeds = rng.normal(size=(npts, net.na))
        seeds[at, a] = np.inf
        got = _gradient(net, X, seeds)[:n * (d0 + 1)].reshape(n, d0 + 1)
        one = np.zeros((1, net.na))
        one[0, a] = 1.0
        f = _gradient(net, X[at:at + 1], one)[:n * (d0 + 1)].reshape(n, d0 + 1)
        s0 = np.sign(f[:, 0]) * np.inf
        assert _same(got[:, 0], s0), a
        for i in range(d0):
            if ts.alpha[a, i] == 0:
                assert _same(got[:, 1 + i], s0), (a, i)
            else:
                se = f[:, 1 + i] - f[:, 0] * X[at, i]
                big = np.abs(se) > 1e-3 * np.max(np.abs(f))  # a sign beyond rounding
                want = np.where(np.sign(se) == np.sign(f[:, 0]), s0, np.nan)
                assert _same(got[big, 1 + i], want[big]), (a, i)
    net.free(); ts.free()


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
@pytest.mark.parametrize("npts", [3, 3000])
def test_first_layer_rows(npts, prec, pin):
    """A row whose seed overflows (an infinite coefficient) has the classes of
    the gradient at that seed; the other slots' rows are finite."""
    ts, dims = api.TableSet(4, 4), [4, 20, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 4), precision=prec)
    X = np.random.default_rng(2).uniform(0.25, 1.0, (npts, 4))
    pin(2, 2)
    a = ts.slot([0, 2, 0, 1])
    rule = api.SeedRule(api.SEED_JROW, [(1.0, 1, False), (np.inf, a, False)])
    rows = api.jacobian_rows(net, X, rule)[0]
    seeds = np.zeros((1, net.na))
    seeds[0, 0], seeds[0, a - 1] = 1.0, np.inf
    for p in (0, npts - 1):
        assert _same(rows[p][:100], _gradient(net, X[p:p + 1], seeds)[:100])
    rule.free(); net.free(); ts.free()


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("d0,k,dims,npts", [(2, 4, [2, 9, 13, 1], 3), (3, 3, [3, 8, 8, 8, 1], 200),
                                            (4, 4, [4, 5, 1], 40)])
def test_one_launch_step(d0, k, dims, npts, value, pin):
    """The one-launch step against the layered kernels, every weight."""
    ts = api.TableSet(d0, k)
    net = api.Net(ts, dims, weights=xavier_weights(dims, 5))
    X = np.random.default_rng(3).uniform(0.25, 1, (npts, d0))
    for a in range(0, net.na, 3):
        seeds = np.random.default_rng(a).normal(size=(npts, net.na))
        seeds[npts // 2, a] = value
        pin(-1, -1)
        api.profile_enable(True)
        api.profile_read()
        got = _gradient(net, X, seeds)
        names = api.profile_read()
        api.profile_enable(False)
        assert "k_point" in names
        pin(2, 2)
        assert _same(got, _gradient(net, X, seeds)), a
    net.free(); ts.free()
