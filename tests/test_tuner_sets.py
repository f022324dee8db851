"""The autotuner's trials belong to a table set: a second network on an equal
set runs none, one on another set or width its own."""
import numpy as np
import pytest

from conftest import xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


def _launches(d0, k, dims, prec, seeds=None):
    """Launches of a new network's first and second step."""
    ts = api.TableSet(d0, k, seeds)
    net = api.Net(ts, dims, weights=xavier_weights(dims, 1), precision=prec)
    g, r = net.grad(), api.SeedRule(api.SEED_HALFSQ)
    X = np.random.default_rng(0).uniform(-1, 1, (3000, d0))
    out = []
    for _ in range(2):
        n0 = api.launch_count()
        g.rule_batch(X, r)
        out.append(api.launch_count() - n0)
    r.free(); g.free(); net.free(); ts.free()
    return out


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
def test_trials_run_once_a_set(prec):
    dims = [5, 112, 112, 1]                  # no other test's width
    first = _launches(5, 3, dims, prec)
    assert first[0] > first[1]               # the trials
    again = _launches(5, 3, dims, prec)
    assert again[0] - again[1] <= first[0] - first[1] - 6  # none of at least two variants,
    assert again[1] == first[1]                            # forward and adjoint, twice each
    # split operands are made once a network; nothing else differs
    assert again[0] - again[1] <= 2
    other = _launches(5, 3, dims, prec, seeds=[[3, 0, 0, 0, 0], [1, 1, 1, 0, 0], [0, 1, 0, 1, 1],
                                               [0, 0, 3, 0, 0], [2, 0, 0, 0, 1], [0, 2, 0, 1, 0],
                                               [0, 0, 1, 2, 0], [0, 0, 0, 0, 3], [1, 0, 1, 0, 1],
                                               [0, 0, 2, 0, 1], [0, 3, 0, 0, 0], [0, 0, 0, 3, 0]])
    wide = _launches(5, 3, [5, 116, 116, 1], prec)
    assert wide[0] - wide[1] > 2 and other[0] >= other[1]
    for row in api.tune_report():
        if row[4] in (112, 116):
            assert row[6] != 0 and len(row[7]) >= 2
