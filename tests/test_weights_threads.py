"""A network used by two host threads in turn, each on its own per-thread
stream (one handle, two streams): what one sets, the other computes with.
Tolerances as in test_weight_copies.py."""
import threading

import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
PER_THREAD = 2  # cudaStreamPerThread


@pytest.mark.parametrize("prec,tol", [(api.PREC_F64, 1e-12), (api.PREC_SPLIT, 1e-5)])
def test_weights_set_by_another_thread(prec, tol):
    import torch
    d0, k, dims, npts = 2, 3, [2, 32, 32, 1], 1500
    ts, ref = api.TableSet(d0, k), po.Tables(d0, k)
    w = xavier_weights(dims, 3)
    net = api.Net(ts, dims, weights=w, precision=prec)
    X = np.random.default_rng(1).uniform(-1, 1, (npts, d0))
    x = torch.tensor(X, device="cuda")
    wd = [torch.tensor(w * f, device="cuda") for f in np.linspace(0.5, 1.5, 6)]
    tm = [torch.zeros((npts, net.na), dtype=torch.float64, device="cuda") for _ in wd]
    torch.cuda.synchronize()
    errs = []

    def run(name, *args):
        try:
            api.call(name, *args)
        except Exception as e:  # reported by the main thread
            errs.append(e)

    for a, b in zip(wd, tm):
        for name, args in (("dnnf90_set_weights_dev", (net.nid, a.data_ptr(), PER_THREAD)),
                           ("dnnf90_forward_dev", (net.nid, net.tid, npts, x.data_ptr(),
                                                   b.data_ptr(), 0, PER_THREAD))):
            t = threading.Thread(target=run, args=(name,) + args)
            t.start()
            t.join()
    torch.cuda.synchronize()
    assert not errs
    for a, b in zip(wd, tm):
        assert rel_err(b.cpu().numpy(), po.grad_batch(ref, dims, a.cpu().numpy(), X)[1]) < tol
    net.free(); ts.free()
