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
