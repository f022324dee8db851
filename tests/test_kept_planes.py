"""Planes kept by a forward, and what rewrites them before the backward asks
for them: a committee's replay and a replay of a caller's own graph, which run
long after the calls that recorded them.  The gradient is always that of the
points and weights of the backward.  Tolerance: FP64 1e-12, split 1e-5 against
the oracle (as in test_committee.py)."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
D0, K, DIMS, NP = 2, 3, [2, 32, 32, 1], 1500  # more points than the one-launch step takes


@pytest.fixture(params=[api.PREC_F64, api.PREC_SPLIT], ids=["f64", "split"])
def kept(request):
    """A network, two sets of points, and the calls a backward is made of."""
    import torch

    class S:
        pass
    s = S()
    s.tol = 1e-12 if request.param == api.PREC_F64 else 1e-5
    s.ts, s.ref = api.TableSet(D0, K), po.Tables(D0, K)
    s.w = xavier_weights(DIMS, 3)
    s.net = api.Net(s.ts, DIMS, weights=s.w, precision=request.param)
    rng = np.random.default_rng(1)
    s.x, s.y = (torch.tensor(rng.uniform(-1, 1, (NP, D0)), device="cuda") for _ in range(2))
    s.seed = torch.tensor(rng.normal(size=(NP, 1, s.net.na)), device="cuda")
    s.rule = api.SeedRule(api.SEED_HALFSQ)
    s.g2 = torch.zeros(s.net.nw, dtype=torch.float64, device="cuda")
    s.st = lambda: torch.cuda.current_stream().cuda_stream

    def forward():
        api.call("dnnf90_forward_dev", s.net.nid, s.net.tid, NP, s.x.data_ptr(), None, 1, s.st())

    def rule_step():
        api.call("dnnf90_grad_rule_dev", s.net.nid, s.net.tid, NP, s.y.data_ptr(), s.rule.rid,
                 s.g2.data_ptr(), None, None, s.st())

    def backward():
        """The gradient at x and the launches it took."""
        g = torch.zeros(s.net.nw, dtype=torch.float64, device="cuda")
        n0 = api.launch_count()
        api.call("dnnf90_backward_dev", s.net.nid, s.net.tid, NP, s.x.data_ptr(),
                 s.seed.data_ptr(), g.data_ptr(), s.st())
        torch.cuda.synchronize()
        return g.cpu().numpy(), api.launch_count() - n0

    def check(g):
        gref = po.grad_batch(s.ref, DIMS, s.w, s.x.cpu().numpy(), kind=po.SEED_GIVEN,
                             seeds=s.seed.cpu().numpy().reshape(NP, -1), want_t=False)[0]
        assert rel_err(g, gref) < s.tol
    s.forward, s.rule_step, s.backward, s.check = forward, rule_step, backward, check
    yield s
    s.rule.free(); s.net.free(); s.ts.free()


def test_kept_planes_save_the_forward(kept):
    kept.forward()
    g, n_kept = kept.backward()
    kept.check(g)
    g, n_again = kept.backward()  # the planes outlive a backward
    kept.check(g)
    kept.rule_step()              # other points' planes
    g, n_recomputed = kept.backward()
    kept.check(g)
    assert n_kept == n_again < n_recomputed


@pytest.mark.parametrize("between", ["batch", "queue", "rows"])
def test_host_calls_between(kept, between):
    """The host entries that write the same work space's planes, through the
    layered kernels (a pinned variant: the one-launch step touches no plane),
    the batch and the rows at the kept points themselves."""
    X = kept.x.cpu().numpy()
    g = kept.net.grad()
    j = api.SeedRule(api.SEED_JROW, [(1.0, 1, False)])
    api.tune_force(0, 2)
    try:
        kept.forward()
        n_kept = kept.backward()[1]
        if between == "batch":
            g.rule_batch(X, kept.rule)
        elif between == "queue":
            for p in range(3):
                g.point(kept.y[p].cpu().numpy(), np.ones(kept.net.na))
            g.read()
        else:
            api.jacobian_rows(kept.net, X[:40], j)
        got, n = kept.backward()
    finally:
        api.tune_force(0, -1)
    kept.check(got)
    assert n > n_kept            # recomputed
    j.free(); g.free()


def test_committee_replay_between(kept):
    import torch
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    step = lambda: api.committee_step([kept.net], [kept.rule], [kept.y], [kept.g2], loss)
    step()                        # builds the graph
    kept.forward()
    step()                        # a replay
    kept.check(kept.backward()[0])


def test_graph_replay_between(kept):
    import torch
    kept.rule_step()              # settles allocations and variant choices
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kept.rule_step()
    kept.forward()
    graph.replay()
    kept.check(kept.backward()[0])
    kept.forward()                # and planes kept after the replay are good again
    _, n = kept.backward()
    kept.rule_step()
    assert n < kept.backward()[1]


def test_forward_captured_and_not_run(kept):
    import torch
    kept.forward()
    kept.rule_step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kept.forward()
    kept.check(kept.backward()[0])  # the planes are those of y
    graph.replay()
    kept.check(kept.backward()[0])


def test_forward_and_backward_in_one_graph(kept):
    import torch
    g = torch.zeros(kept.net.nw, dtype=torch.float64, device="cuda")

    def step():
        g.zero_()
        kept.forward()
        api.call("dnnf90_backward_dev", kept.net.nid, kept.net.tid, NP, kept.x.data_ptr(),
                 kept.seed.data_ptr(), g.data_ptr(), kept.st())
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    n0 = api.launch_count()
    with torch.cuda.graph(graph):
        step()
    n_graph = api.launch_count() - n0
    kept.rule_step()
    kept.x.mul_(0.5)
    graph.replay()
    torch.cuda.synchronize()
    kept.check(g.cpu().numpy())
    kept.rule_step()
    n0 = api.launch_count()
    kept.backward()
    assert n_graph < 2 * (api.launch_count() - n0)
