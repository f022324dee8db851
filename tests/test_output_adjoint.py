"""The output layer's adjoint in each of its forms (block sums or not, loads
ahead or not), at the edges of the widths, slots and points that choose them:
gradient and rows against the oracle.  Tolerances FP64 1e-12, split 1e-5 (as in
test_gpu_parity.py)."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(api.PREC_F64, 1e-12), (api.PREC_SPLIT, 1e-5)])
@pytest.mark.parametrize("d0,k,width,npts", [
    (1, 2, 32, 5), (1, 2, 33, 511), (1, 2, 33, 512), (2, 2, 64, 513), (2, 2, 65, 511),
    (2, 2, 128, 600), (2, 2, 129, 512), (2, 2, 256, 700), (2, 7, 65, 520), (2, 8, 65, 520),
    (3, 3, 40, 9), (2, 8, 200, 3), (2, 2, 260, 30)])
def test_output_adjoint(prec, tol, d0, k, width, npts):
    ts, ref, dims = api.TableSet(d0, k), po.Tables(d0, k), [d0, width, 1]
    w = xavier_weights(dims, 3)
    net = api.Net(ts, dims, weights=w, precision=prec)
    X = np.random.default_rng(npts).uniform(-1, 1, (npts, d0))
    rule, g = api.SeedRule(api.SEED_HALFSQ), net.grad()
    jrule = api.SeedRule(api.SEED_JROW, [(1.0, 1, False), (0.5, net.na, False)])
    api.tune_force(0, 2)  # the layered kernels for small batches too
    try:
        g.rule_batch(X, rule)
        rows = api.jacobian_rows(net, X[:7], jrule)[0]
        gr = net.grad()
        seeds = np.zeros((7, net.na))
        seeds[:, 0] += 1.0
        seeds[:, net.na - 1] += 0.5
        gr.batch(X[:7], seeds)
    finally:
        api.tune_force(0, -1)
    gref = po.grad_batch(ref, dims, w, X, want_t=False)[0]
    m = width * (d0 + 1)
    assert rel_err(g.read()[m:], gref[m:]) < tol and rel_err(g.read(), gref) < tol
    assert rel_err(rows.sum(axis=0), gr.read()) < tol
    for h in (rule, jrule, g, gr, net, ts):
        h.free()
