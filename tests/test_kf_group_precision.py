"""How far grouped and single Kalman updates are from 80-bit arithmetic, where
the rows resemble each other and where they do not, and rows whose own square
overflows."""
import numpy as np
import pytest

from conftest import rel_err
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
DIMS = [3, 32, 32, 1]


@pytest.fixture
def path():
    yield lambda v: api.tune_force(3, v)
    api.tune_force(3, -1)


def _run(w0, rows, xi, p0, lam, lam0, q):
    ts = api.TableSet(DIMS[0], 1)
    net = api.Net(ts, DIMS, weights=w0)
    kf = api.Kalman(net, p0, lam, lam0, False, q, 0.0)
    kf.update_rows(rows, xi)
    out = net.get_weights(), kf.cov()
    kf.free(); net.free(); ts.free()
    return out


def _exact(w0, rows, xi, p0, lam, lam0, q):
    L = np.longdouble
    w, P = w0.astype(L), L(p0) * np.eye(len(w0), dtype=L)
    for r, e in zip(rows.astype(L), xi.astype(L)):
        p = P @ r
        d = L(lam) + r @ p
        w += p * (e / d)
        P -= np.outer(p, p / d)
        P /= L(lam)
        P[np.diag_indices(len(w))] += L(q)
        lam = (lam0 * lam + 1.0) - lam0  # the filter's own sequence, in doubles
    return w, P


def _rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("p0,corr,q", [(0.7, 0.0, 0.0), (100.0, 0.99, 0.0), (100.0, 0.99, 1e-4),
                                       (1e4, 0.9999, 0.0)])
def test_groups_are_as_close_as_single_updates(p0, corr, q, path):
    """Root mean square errors of the weights and of the covariance over three
    draws.  An observation's vector is rounded to doubles three times in a
    group (Y, U and the sum with the covariance), where a single update rounds
    the covariance: at most three times the single updates' error, or one unit
    in the last place."""
    nw = 32 * 4 + 32 * 33 + 33
    err = []
    for seed in range(3):
        rng = np.random.default_rng(seed)
        rows = (np.sqrt(corr) * rng.normal(size=nw) + np.sqrt(1 - corr) * rng.normal(size=(24, nw)))
        xi, w0 = rng.normal(size=24) * 0.1, rng.normal(size=nw) * 0.3
        args = (w0, rows, xi, p0, 0.98, 0.999, q)
        exact = _exact(*args)
        path(0)
        single = _run(*args)
        path(-1)
        group = _run(*args)
        err.append([[_rms(a, e) for a, e in zip(r, exact)] for r in (group, single)])
    group, single = np.sqrt(np.mean(np.square(err), axis=0))
    assert np.all(group <= np.maximum(3 * single, 2.0 ** -52)), (group, single)


def test_rows_whose_square_overflows(path):
    """|j|^2 beyond the largest double with j P j inside it: without process
    noise the update counts on the second alone, as single updates do."""
    nw = 32 * 4 + 32 * 33 + 33
    rng = np.random.default_rng(4)
    rows = rng.normal(size=(9, nw)) * 1e154
    rows[::2] *= 1e-150
    args = (rng.normal(size=nw), rows, rng.normal(size=9), 1e-24, 0.98, 0.999, 0.0)
    path(0)
    w1, P1 = _run(*args)
    path(-1)
    wg, Pg = _run(*args)
    assert np.all(np.isfinite(wg)) and rel_err(wg, w1) < 1e-11 and rel_err(Pg, P1) < 1e-11
