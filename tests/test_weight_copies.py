"""Weights that live on the device between calls: the host copy, the split
operands and the planes kept for a backward follow them in every order of the
calls that read or write them.  Tolerances: FP64 results 1e-12 against the
oracle, weights exact."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
D0, K, DIMS = 2, 3, [2, 32, 32, 1]


def _setup(prec=api.PREC_F64):
    ts, ref = api.TableSet(D0, K), po.Tables(D0, K)
    w = xavier_weights(DIMS, 3)
    X = np.random.default_rng(1).uniform(-1, 1, (70, D0))
    return api.Net(ts, DIMS, weights=w, precision=prec), ts, ref, w, X


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
def test_adam_then_every_reader(prec):
    net, ts, ref, w, X = _setup(prec)
    g, r = net.grad(), api.SeedRule(api.SEED_HALFSQ)
    tol = 1e-12 if prec == api.PREC_F64 else 1e-5
    for step in (1, 2):
        g.zero()
        g.rule_batch(X, r)
        gref = po.grad_batch(ref, DIMS, net.get_weights(), X, want_t=False)[0]
        assert rel_err(g.read(), gref) < tol     # the weights of this step, not the last
        g.adam(1e-2, 0.9, 0.999, 1e-8, len(X), step)
        T = net.eval(X)                          # device weights, host copy not fetched yet
        w2 = net.get_weights()
        assert np.max(np.abs(w2 - w)) > 1e-3
        assert rel_err(T, po.grad_batch(ref, DIMS, w2, X)[1]) < tol
        w = w2
    # one layer set on the host after a device update keeps the others
    n2 = DIMS[1] * (DIMS[0] + 1)
    api.call("dnnf90_net_set_layer", net.nid, 2, api._pd(np.zeros(n2)))
    w3 = net.get_weights()
    assert np.all(w3[:n2] == 0.0) and np.array_equal(w3[n2:], w[n2:])
    r.free(); g.free(); net.free(); ts.free()


def test_set_weights_dev_versions():
    import torch
    net, ts, ref, w, X = _setup()
    st = torch.cuda.current_stream().cuda_stream
    wd = torch.tensor(w * 1.5, device="cuda")
    api.call("dnnf90_set_weights_dev", net.nid, wd.data_ptr(), st)
    assert np.array_equal(net.get_weights(), w * 1.5)
    wd[7] += 0.25
    api.call("dnnf90_set_weights_dev", net.nid, wd.data_ptr(), st)
    assert np.array_equal(net.get_weights(), wd.cpu().numpy())
    net.set_precision(api.PREC_SPLIT)            # its operands from the device weights
    assert rel_err(net.eval(X), po.grad_batch(ref, DIMS, wd.cpu().numpy(), X)[1]) < 1e-5
    s = torch.cuda.Stream()
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr, stream=s):
        rc = api.lib().dnnf90_set_weights_dev(net.nid, wd.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream)
        wd.add_(0.0)
    assert rc == -3
    net.free(); ts.free()


@pytest.mark.parametrize("between", ["nothing", "points", "batch", "queue", "weights"])
def test_kept_planes_follow_points_and_weights(between):
    """A kept forward, then something that makes its planes stale (or not),
    then the backward: always the gradient at the current points and weights."""
    import torch
    net, ts, ref, w, X = _setup()
    st = torch.cuda.current_stream().cuda_stream
    x = torch.tensor(X, device="cuda")
    seed = torch.tensor(np.random.default_rng(2).normal(size=(len(X), 1, net.na)), device="cuda")
    api.call("dnnf90_forward_dev", net.nid, net.tid, len(X), x.data_ptr(), None, 1, st)
    g0 = net.grad()
    if between == "points":
        x.mul_(0.5)                              # the same buffer, other points
    elif between == "batch":
        r = api.SeedRule(api.SEED_HALFSQ)
        g0.rule_batch(X * 0.3, r)
        r.free()
    elif between == "queue":
        g0.point(X[0], np.ones(net.na))
        g0.read()
    elif between == "weights":
        w = w * 0.9
        net.set_weights(w)
    g = torch.zeros(net.nw, dtype=torch.float64, device="cuda")
    n0 = api.launch_count()
    api.call("dnnf90_backward_dev", net.nid, net.tid, len(X), x.data_ptr(), seed.data_ptr(),
             g.data_ptr(), st)
    torch.cuda.synchronize()
    gref = po.grad_batch(ref, DIMS, w, x.cpu().numpy(), kind=po.SEED_GIVEN,
                         seeds=seed.cpu().numpy().reshape(len(X), -1), want_t=False)[0]
    assert rel_err(g.cpu().numpy(), gref) < 1e-12
    assert api.launch_count() > n0
    g0.free(); net.free(); ts.free()
