"""Weight changes around CUDA graph capture: a captured call records no refresh
of the device's copies, so it is refused while they are stale, and neither the
refusal nor an accepted capture disturbs the eager calls around it, on the
capturing stream or another.  Tolerances against the oracle: FP64 1e-12,
split 1e-5 (as in test_weight_copies.py)."""
import numpy as np
import pytest

import pyoracle as po
from conftest import rel_err, xavier_weights
from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
D0, K, NP = 2, 3, 1500
TOL = {api.PREC_F64: 1e-12, api.PREC_SPLIT: 1e-5}


class Case:
    def __init__(self, prec, dims):
        import torch
        self.prec, self.dims = prec, dims
        self.ts, self.ref = api.TableSet(D0, K), po.Tables(D0, K)
        self.net = api.Net(self.ts, dims, weights=xavier_weights(dims, 3), precision=prec)
        self.rule, self.grad = api.SeedRule(api.SEED_HALFSQ), self.net.grad()
        self.X = np.random.default_rng(1).uniform(-1, 1, (NP, D0))
        self.x = torch.tensor(self.X, device="cuda")
        self.g = torch.zeros(self.net.nw, dtype=torch.float64, device="cuda")
        self.stream = torch.cuda.Stream()

    def step(self):
        """The return code of one device step on the current stream."""
        import torch
        return api.lib().dnnf90_grad_rule_dev(
            self.net.nid, self.net.tid, NP, self.x.data_ptr(), self.rule.rid, self.g.data_ptr(),
            None, None, torch.cuda.current_stream().cuda_stream)

    def capture(self):
        """(graph, return code of the captured step)"""
        import torch
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=self.stream):
            self.g.zero_()
            rc = self.step()
        return graph, rc

    def adam(self, istep):
        self.grad.zero()
        self.grad.rule_batch(self.X, self.rule)
        self.grad.adam(1e-2, 0.9, 0.999, 1e-8, NP, istep)

    def check(self):
        """self.g against the oracle at the current weights."""
        import torch
        torch.cuda.synchronize()
        gref = po.grad_batch(self.ref, self.dims, self.net.get_weights(), self.X,
                             want_t=False)[0]
        assert rel_err(self.g.cpu().numpy(), gref) < TOL[self.net.precision]

    def eager(self):
        """Eager steps on the default stream and on the capturing one."""
        import torch
        for s in (torch.cuda.default_stream(), self.stream):
            with torch.cuda.stream(s):
                self.g.zero_()
                assert self.step() == 0
            self.check()

    def free(self):
        self.rule.free(); self.grad.free(); self.net.free(); self.ts.free()


@pytest.mark.parametrize("dims", [[2, 48, 1], [2, 32, 32, 1]])
@pytest.mark.parametrize("change", ["host", "adam", "precision"])
@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
def test_capture_after_a_weight_change(prec, change, dims):
    c = Case(prec, dims)
    assert c.step() == 0          # planes, tables, variant choices
    if change == "host":
        c.net.set_weights(c.net.get_weights() * 1.25)
    elif change == "adam":
        c.adam(1)
    else:
        # planes of the other precision, then weights it has not seen
        c.net.set_precision(api.PREC_SPLIT)
        assert c.step() == 0
        c.net.set_precision(api.PREC_F64)
        c.adam(1)
        c.net.set_precision(api.PREC_SPLIT)
    stale = change == "host" or c.net.precision == api.PREC_SPLIT
    graph, rc = c.capture()
    assert rc == (-3 if stale else 0)
    if stale:
        assert "outside the capture" in api.lib().dnnf90_last_error().decode()
        c.eager()
        graph, rc = c.capture()
        assert rc == 0
    graph.replay()
    c.check()
    c.eager()
    c.free()


def test_capture_waits_for_operands_still_being_made():
    """Weights set on one stream, the step captured on another and replayed."""
    import torch
    c = Case(api.PREC_SPLIT, [2, 32, 32, 1])
    assert c.step() == 0
    other = torch.cuda.Stream()
    for f in (0.5, 1.5):
        wd = torch.tensor(c.net.get_weights() * f, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        api.call("dnnf90_set_weights_dev", c.net.nid, wd.data_ptr(), other.cuda_stream)
        with torch.cuda.graph(graph, stream=c.stream):
            c.g.zero_()
            assert c.step() == 0
        graph.replay()
        c.check()
        c.eager()
    c.free()


@pytest.mark.parametrize("prec", [api.PREC_F64, api.PREC_SPLIT])
def test_adam_step_ends_with_the_update(prec):
    """The weights are written when the call returns, also behind work that
    was on the default stream already, so a replay may follow at once."""
    import torch
    c = Case(prec, [2, 32, 32, 1])
    assert c.step() == 0
    graph, rc = c.capture()
    assert rc == 0
    for istep in (1, 2):
        c.grad.zero()
        c.grad.rule_batch(c.X, c.rule)
        torch.cuda._sleep(20_000_000)  # some 10 ms
        c.grad.adam(1e-2, 0.9, 0.999, 1e-8, NP, istep)
        assert torch.cuda.default_stream().query()
        if prec == api.PREC_SPLIT:     # the operands follow on a call outside the graph
            c.net.eval(c.X[:1])
        with torch.cuda.stream(c.stream):
            graph.replay()
        c.check()
    c.free()
