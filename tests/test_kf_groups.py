"""The grouped Kalman updates of larger filters (eight observations to a pass
over the covariance) against the oracle's observation-by-observation filter,
at the bar the single updates meet: group remainders, the gate and process
noise, the decoupled covariance, a failing observation at every place of a
group, calls of one or two observations in between, and the device entry."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
DENSE, BLOCKS = [3, 32, 32, 1], [2, 84, 80, 1]     # 741 tiles; single updates on its 85-wide blocks
WIDE = [2, 45, 46, 1]                              # 2298 weights: row blocks of several items


def _rows(nw, nobs, seed):
    rng = np.random.default_rng(seed)
    return (rng.normal(size=(nobs, nw)) / np.sqrt(nw), rng.normal(size=nobs) * 2.0,
            rng.uniform(0.5, 1.5, nobs))


def _pair(dims, dec, q, gate):
    nw = po.weight_count(dims)
    w0 = np.random.default_rng(5).normal(size=nw) * 0.1
    ts = api.TableSet(dims[0], 1)
    net = api.Net(ts, dims, weights=w0)
    kf = api.Kalman(net, 0.7, 0.98, 0.9987, dec, q, gate)
    return kf, net, ts, po.Kalman(dims, 0.7, 0.98, 0.9987, dec, q, gate), w0.copy()


def _check(kf, net, ref, wref):
    lam, ng = kf.state()
    assert ng == ref.ngated.value and abs(lam - ref.lam) <= 1e-15
    assert rel_err(net.get_weights(), wref) < 1e-11, rel_err(net.get_weights(), wref)
    P = kf.cov()
    assert rel_err(P.reshape(-1), ref.P) < 1e-11, rel_err(P.reshape(-1), ref.P)
    if P.ndim == 2:
        assert np.array_equal(P, P.T)


@pytest.mark.parametrize("dims,dec,q,gate", [
    (DENSE, False, 0.0, 0.0), (DENSE, False, 1e-4, 1.0), (BLOCKS, True, 0.0, 0.0),
    (BLOCKS, True, 1e-4, 1.0), (WIDE, False, 1e-4, 1.0)])
@pytest.mark.parametrize("nobs", [3, 8, 9, 21])
def test_matches_the_oracle(dims, dec, q, gate, nobs):
    kf, net, ts, ref, wref = _pair(dims, dec, q, gate)
    rows, xi, sc = _rows(net.nw, nobs, nobs)
    kf.update_rows(rows, xi, sc)
    for r, e, s in zip(rows, xi, sc):
        ref.update(wref, r, e, s)
    if gate:
        assert ref.ngated.value > 0
    _check(kf, net, ref, wref)
    kf.free(); net.free(); ts.free()


def test_calls_of_every_length_in_turn(monkeypatch):
    """Grouped and single calls alternate, and a staging area of ten rows cuts
    a call into chunks of which the last has one observation."""
    kf, net, ts, ref, wref = _pair(DENSE, False, 1e-5, 0.0)
    rows, xi, sc = _rows(net.nw, 40, 2)
    k = 0
    for m in (1, 5, 2, 8, 1, 3):
        kf.update_rows(rows[k:k + m], xi[k:k + m], sc[k:k + m])
        k += m
    monkeypatch.setenv("DNNF90_KF_STAGE_KB", str(net.nw * 8 * 10 // 1024 + 1))
    kf.update_rows(rows[k:41], xi[k:41], sc[k:41])
    for r, e, s in zip(rows, xi, sc):
        ref.update(wref, r, e, s)
    _check(kf, net, ref, wref)
    kf.free(); net.free(); ts.free()


@pytest.mark.parametrize("bad", [0, 1, 7, 8, 11])
def test_stops_at_a_nonpositive_denominator(bad):
    kf, net, ts, ref, wref = _pair(DENSE, False, 0.0, 0.0)
    rows, xi, sc = _rows(net.nw, 20, 7)
    rows[bad, 17] = np.nan
    with pytest.raises(api.Dnnf90Error):
        kf.update_rows(rows, xi, sc)
    assert api.lib().dnnf90_kf_status(kf.kid) == bad + 1
    for k in range(bad):
        ref.update(wref, rows[k], xi[k], sc[k])
    _check(kf, net, ref, wref)
    kf.update_rows(rows[bad + 1:], xi[bad + 1:], sc[bad + 1:])
    assert api.lib().dnnf90_kf_status(kf.kid) == 0
    for k in range(bad + 1, 20):
        ref.update(wref, rows[k], xi[k], sc[k])
    _check(kf, net, ref, wref)
    kf.free(); net.free(); ts.free()


def test_device_entry_and_graph_replay():
    """The device entry, called and replayed from a CUDA graph, gives the
    host entry's filter bit for bit."""
    import torch
    kf, net, ts, _, w0 = _pair(DENSE, False, 1e-4, 1.0)
    rows, xi, sc = _rows(net.nw, 11, 9)
    kf.update_rows(rows, xi, sc)
    w1, P1 = net.get_weights(), kf.cov()
    dev = torch.device("cuda", 0)
    r, x, c = (torch.tensor(a, device=dev) for a in (rows, xi, sc))
    for graph in (False, True):
        k2 = api.Kalman(net, 0.7, 0.98, 0.9987, False, 1e-4, 1.0)
        w = torch.tensor(w0, device=dev)

        def call(st):
            api.call("dnnf90_kf_update_rows_dev", k2.kid, 11, r.data_ptr(), x.data_ptr(),
                     c.data_ptr(), w.data_ptr(), st.cuda_stream)
        if graph:
            s = torch.cuda.Stream(dev)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                call(torch.cuda.current_stream(dev))
            g.replay()
            torch.cuda.synchronize(dev)
            assert api.lib().dnnf90_kf_status(k2.kid) == 0
        else:
            call(torch.cuda.current_stream(dev))
        assert np.array_equal(w.cpu().numpy(), w1) and np.array_equal(k2.cov(), P1)
        k2.free()
    kf.free(); net.free(); ts.free()
