"""The first-layer gradient of the split path: how far its sums over the slots
run in FP32, and its error against FP64."""
import numpy as np
import pytest

from conftest import xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


def _backward(net, x, seed):
    import torch
    g = torch.zeros(net.nw, dtype=torch.float64, device="cuda")
    api.call("dnnf90_backward_dev", net.nid, net.tid, x.shape[0], x.data_ptr(), seed.data_ptr(),
             g.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return g.cpu().numpy()


@pytest.mark.parametrize("d0,k,lost", [(4, 7, 7), (4, 5, 3), (3, 6, 0)])
def test_a_large_slot_swallows_no_more_than_its_run(d0, k, lost):
    """Weights of one make every slot of the top degree count alike.  The first
    holds B and the last -B, each other 1, half an ulp of B in FP32: what is
    added to B in FP32 is lost, so the sum misses at most the other slots of
    the two runs that hold B (runs of |A| / 32 slots in whole groups of four,
    sums in FP64 where that is less than a group), beside the FP32 rounding of
    s^(k+1) and of the monomials (4 u each)."""
    import torch
    B, npts, n = 2.0 ** 24, 20000, 32
    ts = api.TableSet(d0, k)
    w = np.ones(n * (d0 + 1) + n + 1)
    w[:n * (d0 + 1):d0 + 1] = 0.5
    net = api.Net(ts, [d0, n, 1], weights=w, precision=api.PREC_SPLIT)
    top = np.nonzero(ts.alpha.sum(axis=1) == k)[0]
    seed = np.zeros((1, net.na))
    seed[0, top] = 1.0
    seed[0, top[0]], seed[0, top[-1]] = B, -B
    x = torch.zeros((npts, d0), dtype=torch.float64, device="cuda")
    sd = torch.tensor(np.repeat(seed[None], npts, axis=0), device="cuda")
    g = _backward(net, x, sd)[:n * (d0 + 1):d0 + 1]
    net.set_precision(api.PREC_F64)
    ref = _backward(net, x, sd)[:n * (d0 + 1):d0 + 1]
    ones = len(top) - 2
    assert np.all(np.abs(g / ref - 1.0) <= 2 * lost / ones + 8 * 2.0 ** -24)
    net.free(); ts.free()


@pytest.mark.parametrize("d0,k,n,npts", [(4, 7, 33, 3001), (4, 3, 20, 70), (2, 6, 8, 5000),
                                         (1, 9, 16, 999), (8, 2, 64, 1), (6, 4, 40, 4097)])
def test_gradient_against_fp64(d0, k, n, npts):
    """Both forms of the sums (runs in FP32, FP64 throughout), ragged tiles and
    points.  Each product carries the roundings of Tb, of s and of a monomial
    (its k factors and a!), each a unit roundoff of FP32, and a run of at most
    16 slots as many again; the bound is on the sum of magnitudes, bounded here
    by that of the gradient at seeds of one sign over the points."""
    import torch
    ts = api.TableSet(d0, k)
    dims = [d0, n, 1]
    w = xavier_weights(dims, 5)
    rng = np.random.default_rng(n)
    x = torch.tensor(rng.uniform(-1, 1, (npts, d0)), device="cuda")
    # seeds that fall with the order, so that no order swamps the others
    sd = torch.tensor(rng.normal(size=(npts, 1, ts.na)) / 4.0 ** ts.alpha.sum(axis=1), device="cuda")
    net = api.Net(ts, dims, weights=w, precision=api.PREC_SPLIT)
    g = _backward(net, x, sd)
    net.set_precision(api.PREC_F64)
    ref = _backward(net, x, sd)
    m = n * (d0 + 1)
    assert np.max(np.abs(g[:m] - ref[:m])) <= (k + 20) * 2.0 ** -24 * npts ** 0.5 * np.max(np.abs(ref[:m]))
    net.free(); ts.free()


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
@pytest.mark.parametrize("d0,k,n,npts", [(4, 4, 33, 37), (4, 7, 16, 5), (3, 6, 8, 70)])
def test_rows_add_up_to_the_gradient(prec, d0, k, n, npts):
    """Jacobian rows of more than 36 slots (the same kernel, a point at a
    time): their sum is the gradient at a residual's seeds."""
    import torch
    ts = api.TableSet(d0, k)
    dims = [d0, n, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 6), precision=prec)
    terms = [(1.0 / (1 + s), s + 1, False) for s in range(0, net.na, 3)]
    rule = api.SeedRule(api.SEED_JROW, terms)
    X = np.random.default_rng(n).uniform(-1, 1, (npts, d0))
    api.tune_force(0, 2)  # the layered kernels in FP64 too
    try:
        rows = api.jacobian_rows(net, X, rule)[0]
        seed = np.zeros((npts, 1, net.na))
        for c, s, _ in terms:
            seed[:, 0, s - 1] += c
        g = _backward(net, torch.tensor(X, device="cuda"), torch.tensor(seed, device="cuda"))
    finally:
        api.tune_force(0, -1)
    u = 2.0 ** -24 if prec == api.PREC_SPLIT else 2.0 ** -52
    scale = np.sum(np.abs(rows), axis=0)
    assert np.all(np.abs(rows.sum(axis=0) - g) <= (k + 2 * net.na + npts) * u * np.max(scale))
    rule.free(); net.free(); ts.free()


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
@pytest.mark.parametrize("d0,k,n", [(4, 3, 32), (2, 7, 33), (1, 5, 3), (3, 2, 129), (8, 1, 20),
                                    (4, 3, 5)])
def test_small_set_rows_have_one_rounding(prec, d0, k, n):
    """A row of a set of at most 36 slots has the same bits alone, among few
    points and among many (the block's warps share a point's slots or not)."""
    ts = api.TableSet(d0, k)
    dims = [d0, n, 1]
    net = api.Net(ts, dims, weights=xavier_weights(dims, 6), precision=prec)
    rule = api.SeedRule(api.SEED_JROW, [(1.0, net.na, False), (0.3, 1, False)])
    X = np.random.default_rng(n).uniform(-1, 1, (40000, d0))
    api.tune_force(0, 4)
    try:
        many = api.jacobian_rows(net, X, rule)[0]
        for npts in (1, 2, 37, 700):
            assert np.array_equal(api.jacobian_rows(net, X[:npts], rule)[0], many[:npts]), npts
    finally:
        api.tune_force(0, -1)
    rule.free(); net.free(); ts.free()
