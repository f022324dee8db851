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


def test_a_filter_of_single_observations_has_no_group_buffers():
    """The groups' buffers (some 60 MB at 17025 weights) come with the first
    call that groups, which may be one in a capture."""
    import torch
    dims = [2, 128, 128, 1]
    ts = api.TableSet(2, 1)
    nw = 128 * 3 + 128 * 129 + 129
    rng = np.random.default_rng(0)
    net = api.Net(ts, dims, weights=rng.normal(size=nw) * 0.1)
    rows = torch.tensor(rng.normal(size=(9, nw)) * 0.05, device="cuda")
    xi = torch.tensor(rng.normal(size=9), device="cuda")
    w0 = torch.tensor(rng.normal(size=nw), device="cuda")
    api.Kalman(net, 0.5, 0.98, 0.99).free()          # whatever a first filter loads

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    def update(kf, nobs, w):
        api.call("dnnf90_kf_update_rows_dev", kf.kid, nobs, rows.data_ptr(), xi.data_ptr(), None,
                 w.data_ptr(), torch.cuda.current_stream().cuda_stream)

    tb = (nw + 31) // 32
    cov = tb * (tb + 1) // 2 * 32 * 32 * 8 + tb * tb * 32 * 8  # the tiles and their partial sums
    base = used()
    kf = api.Kalman(net, 0.5, 0.98, 0.99)
    w = w0.clone()
    update(kf, 1, w)
    update(kf, 2, w)
    assert used() - base <= cov + (24 << 20)
    before = used()
    update(kf, 3, w)
    assert used() - before >= 30 << 20
    kf.free()
    # a capture before the first grouped call, and the same calls outside one
    out = []
    for captured in (True, False):
        kf = api.Kalman(net, 0.5, 0.98, 0.99)
        w = w0.clone()
        if captured:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                update(kf, 9, w)
            graph.replay()
            torch.cuda.synchronize()
        else:
            update(kf, 9, w)
        update(kf, 9, w)
        out.append(w.cpu().numpy())
        kf.free()
    assert np.array_equal(out[0], out[1])
    net.free(); ts.free()
