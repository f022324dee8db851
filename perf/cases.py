"""The work a user of this framework has it do, as measurable cases.

Each case is one pass through the public entry points (dnnf90_b200.api,
dnnf90_b200.autograd) in the way a program calls them: field evaluation from
host points, a training epoch of the host-side trainer, a device-resident
collocation step, a PINN step through torch autograd, a committee of
networks, a damped natural-gradient step and the extended Kalman filter.
Networks, table sets and residuals are those of the repository's benchmark
and tests: dense sets up to D0 = 4, K = 7, the KdV closure and the heat
closure, tanh networks of 8 to 256 neurons a layer.

``exact`` restates every case in plain torch, in 64 bits: a truncated
multivariate Taylor series of the network and its reverse sweep.
"""
import math

import numpy as np
import torch

from dnnf90_b200 import api
from dnnf90_b200.autograd import hod

DEV = "cuda"
SETS = {"dense": None, "kdv": [[0, 1], [1, 0], [3, 0]],
        "heat": [[1, 0, 0], [0, 2, 0], [0, 0, 2]], "value": [[0]]}
BOX = {"kdv": ([-10.0, 0.0], [10.0, 1.0]), "heat": ([0.0] * 3, [1.0] * 3)}
ADAM = (1e-3, 0.9, 0.999, 1e-8)
KF = (0.01, 0.98, 0.9987)          # p0, initial lambda, forgetting schedule


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a host program (a plotting loop, a Fortran or C caller) asks for every
        # mixed partial up to order 7 at one point: the smallest call, all latency
        dict(name="eval_point", kind="eval", set="dense", d0=4, k=7, width=8, hidden=2, npts=1,
             prec=0),
        # the solution and its derivatives up to order 2 over a field, host to host
        dict(name="eval_field", kind="eval", set="dense", d0=3, k=2, width=64, hidden=2,
             npts=100000, prec=0),
        # an epoch of the host-side trainer on the order-7 problem: gradient of a
        # mini-batch, then Adam; small network, launches and host work count
        dict(name="epoch_small", kind="epoch", set="dense", d0=4, k=7, width=8, hidden=2,
             npts=300, prec=0),
        # the plain method: 4-32-32-1, every partial up to order 3, 1024 points
        dict(name="dense_k3", kind="epoch", set="dense", d0=4, k=3, width=32, hidden=2,
             npts=1024, prec=0),
        # a KdV PINN step through torch autograd, FP64
        dict(name="kdv_f64", kind="autograd", set="kdv", d0=2, k=3, width=64, hidden=3,
             npts=16384, prec=0),
        # the same step in split precision with FP32 parameters
        dict(name="kdv_split", kind="autograd", set="kdv", d0=2, k=3, width=64, hidden=3,
             npts=16384, prec=1),
        # the order-7 residual over 65536 device-resident points, split precision:
        # the largest training step
        dict(name="zk7_split", kind="colloc", set="dense", d0=4, k=7, width=128, hidden=3,
             npts=65536, prec=1),
        # the same residual in FP64 on a ragged share of the points
        dict(name="zk7_f64", kind="colloc", set="dense", d0=4, k=7, width=128, hidden=3,
             npts=8191, prec=0),
        # uneven committee: independent networks trained as one step
        dict(name="committee", kind="committee", nets=6, most=12000, pick=20260804),
        # damped natural-gradient step of the heat residual, 4481 weights, 4096
        # points, the metric from split-precision products
        dict(name="ngd_heat", kind="ngd", set="heat", d0=3, k=2, width=64, hidden=2, npts=4096,
             prec=1, route="primal", mu=1e-3),
        # a filter pass over collocation points: the row, residual and update of
        # each point at the weights the previous one left
        dict(name="kalman_pass", kind="kf_pass", set="heat", d0=3, k=2, width=32, hidden=2,
             npts=32),
        # rank-one updates of the dense covariance of a 17025-weight network
        dict(name="kalman_dense", kind="kf_rows", d0=2, k=1, width=128, hidden=2, npts=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nslot(d0, k):
    return math.comb(d0 + k, k)


def draw(rng):
    kind = rng.choice(["eval", "epoch", "colloc", "colloc", "autograd", "autograd", "ngd",
                       "kf_pass", "kf_rows", "committee"])
    if kind in ("eval", "epoch", "colloc"):
        d0, k = rng.randint(2, 4), rng.randint(2, 7)
        width = rng.choice([8, 20, 32, 48, 64, 100, 128] if kind != "colloc"
                           else [32, 48, 64, 128, 256])
        hidden = rng.randint(2, 3 if kind != "colloc" else 4)
        per = _nslot(d0, k) * width * hidden
        if kind == "eval":
            npts, prec = _log(rng, 1, min(100000, 1 + 200000000 // per)), 0
        elif kind == "epoch":
            npts, prec = _log(rng, 10, min(4096, 10 + 60000000 // per)), 0
        else:
            prec = rng.choice([0, 1, 1])
            most = (8000000000 if prec else 1000000000) // per
            npts = _log(rng, 500, max(501, min(65536, most)))
        return dict(kind=kind, set="dense", d0=d0, k=k, width=width, hidden=hidden, npts=npts,
                    prec=prec)
    if kind == "autograd":
        name = rng.choice(["kdv", "heat"])
        return dict(kind=kind, set=name, d0=len(SETS[name][0]), k=3 if name == "kdv" else 2,
                    width=rng.choice([20, 32, 48, 64, 100, 128]), hidden=rng.randint(2, 4),
                    npts=_log(rng, 1000, 65536), prec=rng.choice([0, 1]))
    if kind == "ngd":
        return dict(kind=kind, set="heat", d0=3, k=2, width=rng.choice([16, 24, 32, 48, 56, 64]),
                    hidden=2, npts=_log(rng, 256, 4096), prec=rng.choice([0, 0, 1]),
                    route=rng.choice(["primal", "dual"]), mu=1e-3)
    if kind == "kf_pass":
        name = rng.choice(["heat", "kdv"])
        return dict(kind=kind, set=name, d0=len(SETS[name][0]), k=3 if name == "kdv" else 2,
                    width=rng.choice([16, 20, 32, 40]), hidden=rng.randint(1, 2),
                    npts=rng.randint(8, 32))
    if kind == "kf_rows":
        return dict(kind=kind, d0=rng.randint(2, 4), k=1,
                    width=rng.choice([32, 48, 64, 96, 120, 128]), hidden=2,
                    npts=rng.randint(8, 32))
    return dict(kind=kind, nets=rng.randint(2, 6), most=_log(rng, 2000, 12000),
                pick=rng.randrange(1 << 30))


def _members(case):
    """The committee's draw: widths, depths, sets and point counts."""
    r = np.random.default_rng(case["pick"])
    out = []
    for _ in range(case["nets"]):
        width = int(r.choice([32, 64, 128, 256]))
        hidden, d0, k = int(r.integers(2, 5)), int(r.integers(2, 5)), int(r.integers(2, 8))
        most = min(case["most"], max(1000, 2000000000 // (_nslot(d0, k) * width * hidden)))
        npts = int(np.exp(r.uniform(np.log(1000.0), np.log(max(most, 1001)))))
        out.append(dict(set="dense", d0=d0, k=k, width=width, hidden=hidden, npts=npts, prec=1))
    return out


def _dims(c):
    return [c["d0"]] + [c["width"]] * c["hidden"] + [1]


def _alpha(c):
    """The carried multi-indices in the library's slot order: by degree, then
    in combinations-with-replacement order, restricted to the closure."""
    d0, k, seeds = c["d0"], c["k"], SETS[c.get("set", "dense")]
    out = []

    def rec(v, left, cur):
        if left == 0:
            if seeds is None or any(all(x <= y for x, y in zip(cur, s)) for s in seeds):
                out.append(tuple(cur))
            return
        for j in range(v, d0):
            nxt = list(cur)
            nxt[j] += 1
            rec(j, left - 1, nxt)

    for p in range(k + 1):
        rec(0, p, [0] * d0)
    return out


def _terms(c, alpha):
    """(coefficient, 1-based slot, times u) of the residual."""
    at = {a: i + 1 for i, a in enumerate(alpha)}
    if c["set"] == "kdv":            # u_t + 6 u u_x + u_xxx
        return [(1.0, at[(0, 1)], 0), (6.0, at[(1, 0)], 1), (1.0, at[(3, 0)], 0)]
    if c["set"] == "heat":           # u_t - (u_xx + u_yy)
        return [(1.0, at[(1, 0, 0)], 0), (-1.0, at[(0, 2, 0)], 0), (-1.0, at[(0, 0, 2)], 0)]
    top = [(1.0, i + 1, 0) for i, a in enumerate(alpha) if sum(a) == c["k"]]
    e = [0] * c["d0"]                # every top-order derivative + u u_x
    e[min(1, c["d0"] - 1)] = 1
    return top + [(1.0, at[tuple(e)], 1)]


def _weights(dims, r):
    """Xavier-normal weights and small biases, flat layer layout."""
    out = []
    for m, n in zip(dims[:-1], dims[1:]):
        w = np.empty((n, m + 1))
        w[:, 0] = r.normal(0.0, 0.1, n)
        w[:, 1:] = r.normal(0.0, math.sqrt(2.0 / (m + n)), (n, m))
        out.append(w.reshape(-1))
    return np.concatenate(out)


def _points(c, r):
    lo, hi = BOX.get(c["set"], ([-1.0] * c["d0"], [1.0] * c["d0"]))
    return r.uniform(lo, hi, (c["npts"], c["d0"]))


def _rows(c, nw, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rows = torch.randn((c["npts"], nw), dtype=torch.float64, device=DEV, generator=g)
    xi = torch.randn(c["npts"], dtype=torch.float64, device=DEV, generator=g)
    return rows.div_(math.sqrt(nw)), xi


# ------------------------------------------------------------------ prepare and run
class State:
    """What a program holds between calls: handles, weights, points."""

    def __init__(self, **kw):
        self.held = []
        self.__dict__.update(kw)

    def keep(self, h):
        self.held.append(h)
        return h

    def __del__(self):
        try:
            torch.cuda.synchronize()
            for h in reversed(self.held):
                h.free()
        except Exception:
            pass


def _net(s, c, w):
    ts = s.keep(api.TableSet(c["d0"], c["k"], SETS[c.get("set", "dense")]))
    return s.keep(api.Net(ts, _dims(c), weights=w, precision=c.get("prec", 0)))


def prepare(case, seed):
    c = dict(case)
    r = np.random.default_rng(seed)
    s = State(c=c, kind=c["kind"])
    if s.kind == "committee":
        s.rule = s.keep(api.SeedRule(api.SEED_HALFSQ))
        s.nets, s.xs, s.grads = [], [], []
        for m in _members(c):
            w = _weights(_dims(m), r)
            s.nets.append(_net(s, m, w))
            s.xs.append(torch.tensor(_points(m, r), device=DEV))
            s.grads.append(torch.zeros(len(w), dtype=torch.float64, device=DEV))
        s.loss = torch.zeros(len(s.nets), dtype=torch.float64, device=DEV)
        return s
    w = _weights(_dims(c), r)
    s.net = _net(s, c, w)
    nw = s.net.nw
    if s.kind == "kf_rows":
        s.rows, s.xi = _rows(c, nw, seed)
        s.w = torch.tensor(w, device=DEV)
        s.kf = s.keep(api.Kalman(s.net, *KF))
        return s
    x = _points(c, r)
    alpha = _alpha(c)
    if s.kind == "kf_pass":
        s.x = x
        s.rule = s.keep(api.SeedRule(api.SEED_JROW, _terms(c, alpha)))
        s.kf = s.keep(api.Kalman(s.net, *KF))
    elif s.kind == "eval":
        s.x = x[0] if c["npts"] == 1 else x
    elif s.kind == "epoch":
        s.x = x
        s.rule = s.keep(api.SeedRule(api.SEED_HALFSQ) if c["k"] <= 3
                        else api.SeedRule(api.SEED_PINN, _terms(c, alpha)))
        s.grad = s.keep(s.net.grad())
        s.step = 0
    elif s.kind == "autograd":
        s.x = torch.tensor(x, device=DEV)
        s.w = torch.tensor(w, device=DEV, dtype=torch.float32 if c["prec"] else torch.float64)
        s.w.requires_grad_(True)
        s.terms = _terms(c, alpha)
    else:
        s.x = torch.tensor(x, device=DEV)
        terms = _terms(c, alpha)
        s.rule = s.keep(api.SeedRule(api.SEED_PINN, terms))
        s.g = torch.zeros(nw, dtype=torch.float64, device=DEV)
        s.loss = torch.zeros(1, dtype=torch.float64, device=DEV)
        if s.kind == "ngd":
            s.jrow = s.keep(api.SeedRule(api.SEED_JROW, terms))
            s.rows = torch.empty((c["npts"], nw), dtype=torch.float64, device=DEV)
            if c["route"] == "primal":
                s.G = torch.empty((nw, nw), dtype=torch.float64, device=DEV)
            s.u = torch.empty(nw, dtype=torch.float64, device=DEV)
    return s


def _colloc(s, st):
    s.g.zero_()
    s.loss.zero_()
    api.call("dnnf90_grad_rule_dev", s.net.nid, s.net.tid, s.x.shape[0], s.x.data_ptr(),
             s.rule.rid, s.g.data_ptr(), s.loss.data_ptr(), None, st)


def run(s):
    c = s.c
    if s.kind == "eval":
        return s.net.eval(s.x)
    if s.kind == "epoch":
        s.step += 1
        s.grad.zero()
        loss = s.grad.rule_batch(s.x, s.rule)
        g = s.grad.read()
        s.grad.adam(*ADAM, c["npts"], s.step)
        return {"loss": np.float64(loss), "grad": g, "w": s.net.get_weights()}
    if s.kind == "autograd":
        s.w.grad = None
        t = hod(s.x, s.w, s.net)[:, 0, :].to(s.w.dtype)
        u = t[:, 0]
        res = 0.0
        for co, slot, nl in s.terms:
            v = t[:, slot - 1]
            res = res + co * (u * v if nl else v)
        loss = 0.5 * (res * res).sum()
        loss.backward()
        return {"loss": loss.detach(), "grad": s.w.grad, "res": res.detach()}
    if s.kind == "kf_pass":
        s.kf.pass_points(s.x, s.rule)
        lam, _ = s.kf.state()
        return {"w": s.net.get_weights(), "lam": np.float64(lam)}
    st = torch.cuda.current_stream().cuda_stream
    if s.kind == "kf_rows":
        api.call("dnnf90_kf_update_rows_dev", s.kf.kid, c["npts"], s.rows.data_ptr(),
                 s.xi.data_ptr(), None, s.w.data_ptr(), st)
        return {"w": s.w}
    if s.kind == "committee":
        api.committee_step(s.nets, [s.rule] * len(s.nets), s.xs, s.grads, s.loss)
        # the split path's planes are FP32: the optimizer of each member keeps
        # FP32 parameters and takes FP32 gradients
        return {"loss": s.loss.float(), "grads": [g.float() for g in s.grads]}
    _colloc(s, st)
    if s.kind == "colloc":
        # split precision: FP32 planes, and FP32 parameters on the caller's side
        return ({"loss": s.loss.float(), "grad": s.g.float()} if c["prec"]
                else {"loss": s.loss, "grad": s.g})
    api.call("dnnf90_jrow_dev", s.net.nid, s.net.tid, c["npts"], s.x.data_ptr(), s.jrow.rid,
             s.rows.data_ptr(), None, st)
    nw, n = s.net.nw, c["npts"]
    if c["route"] == "dual":
        api.call("dnnf90_ngd_step_dual_dev", n, nw, s.rows.data_ptr(), s.g.data_ptr(), n,
                 c["mu"], s.u.data_ptr(), st)
    else:
        api.call("dnnf90_ngd_gram_dev", n, nw, s.rows.data_ptr(), c["prec"], s.G.data_ptr(), st)
        api.call("dnnf90_ngd_solve_dev", nw, s.G.data_ptr(), s.g.data_ptr(), n, c["mu"],
                 s.u.data_ptr(), st)
    if c["prec"]:
        return {"u": s.u.float(), "grad": s.g.float(), "loss": s.loss.float()}
    return {"u": s.u, "grad": s.g, "loss": s.loss}


# ------------------------------------------------------------------ work
def _sweep_work(c, train, out_bytes):
    """Points and weights read, results written; the layer products and one
    multiply-add per pair of carried indices, neuron and sweep."""
    na, dims, n = len(_alpha(c)), _dims(c), c["npts"]
    hid = c["width"] * c["hidden"]
    gemm = 2.0 * na * sum(a * b for a, b in zip(dims[1:-1], dims[2:]))
    pairs = float(len(_Series(c, "cpu").pairs[0])) * hid * 2.0
    return {"bytes": n * c["d0"] * 8.0 + 8.0 * sum((a + 1) * b for a, b in zip(dims[:-1], dims[1:]))
            + out_bytes, "flops": n * (3.0 if train else 1.0) * (gemm + pairs)}


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind == "committee":
        parts = [_sweep_work(m, True, 8.0 * _nw(m)) for m in _members(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    nw = _nw(c)
    if kind == "kf_rows":
        # the packed triangle of the covariance read and written at every update
        return {"bytes": c["npts"] * 8.0 * nw * (nw + 2), "flops": c["npts"] * 4.0 * nw * nw}
    if kind == "kf_pass":
        w = _sweep_work(c, True, 8.0 * nw)
        return {"bytes": w["bytes"] + c["npts"] * 8.0 * nw * (nw + 2),
                "flops": w["flops"] + c["npts"] * 4.0 * nw * nw}
    if kind == "eval":
        return _sweep_work(c, False, 8.0 * c["npts"] * len(_alpha(c)))
    w = _sweep_work(c, True, 8.0 * nw)
    if kind == "ngd":
        # the rows written and read, the metric (or Gram matrix) and its factor
        n, m = float(c["npts"]), float(nw if c["route"] == "primal" else c["npts"])
        w["bytes"] += 16.0 * n * nw + 8.0 * m * m
        w["flops"] += n * nw * m + m ** 3 / 3.0
    return w


def _nw(c):
    d = _dims(c)
    return sum((a + 1) * b for a, b in zip(d[:-1], d[1:]))


# ------------------------------------------------------------------ exact values
class _Series:
    """Truncated multivariate Taylor arithmetic over the carried set: arrays
    [na][...] of coefficients d^a f / a!."""

    def __init__(self, c, dev):
        al = _alpha(c)
        at = {a: i for i, a in enumerate(al)}
        self.al, self.na = al, len(al)
        self.deg = [sum(a) for a in al]
        ib, ig, ia = [], [], []
        for b in al:
            for g in al:
                a = tuple(x + y for x, y in zip(b, g))
                if a in at:
                    ib.append(at[b])
                    ig.append(at[g])
                    ia.append(at[a])
        self.pairs = (ib, ig, ia)
        fact = [math.prod(math.factorial(x) for x in a) for a in al]
        if dev != "cpu":
            self.fact = torch.tensor(fact, dtype=torch.float64, device=dev)
            t = torch.tensor
            self.all = tuple(t(v, device=dev) for v in self.pairs)
            self.by = []
            for p in range(1, c["k"] + 1):
                sel = [i for i in range(len(ia)) if self.deg[ia[i]] == p]
                eul = [i for i in sel if self.deg[ib[i]] > 0]
                self.by.append((
                    t([i for i in range(self.na) if self.deg[i] == p], device=dev),
                    tuple(t([v[i] for i in eul], device=dev) for v in self.pairs),
                    t([float(self.deg[ib[i]]) / p for i in eul], dtype=torch.float64, device=dev),
                    tuple(t([v[i] for i in sel], device=dev) for v in self.pairs)))

    def tanh(self, s):
        """t = tanh(s) and u = 1 - t^2, degree by degree: |a| t_a = sum |b|
        s_b u_(a-b) (Euler's relation), u_a = -sum t_b t_(a-b)."""
        t, u = torch.zeros_like(s), torch.zeros_like(s)
        t[0] = torch.tanh(s[0])
        u[0] = 1.0 - t[0] * t[0]
        for slots, (ib, ig, ia), f, (jb, jg, ja) in self.by:
            if len(slots) == 0:
                continue
            t.index_add_(0, ia, s[ib] * u[ig] * f.view(-1, 1, 1))
            u.index_add_(0, ja, t[jb] * t[jg], alpha=-1.0)
        return t, u

    def adjoint(self, tb, u):
        """d/ds of <tb, t(s)>: sb_b = sum tb_(b+g) u_g."""
        ib, ig, ia = self.all
        sb = torch.zeros_like(tb)
        sb.index_add_(0, ib, tb[ia] * u[ig])
        return sb


def _layers(c, w):
    d, out, off = _dims(c), [], 0
    for m, n in zip(d[:-1], d[1:]):
        out.append(w[off:off + n * (m + 1)].view(n, m + 1))
        off += n * (m + 1)
    return out


def _forward(se, c, w, x):
    """Planes of a chunk of points: inputs of every layer, u of the hidden
    ones, and the output derivatives [P][na]."""
    L = _layers(c, w)
    t = torch.zeros((se.na, x.shape[0], c["d0"]), dtype=torch.float64, device=x.device)
    t[0] = x
    for j in range(c["d0"]):
        e = tuple(int(i == j) for i in range(c["d0"]))
        if e in se.al:
            t[se.al.index(e), :, j] = 1.0
    ins, us = [], []
    for l, W in enumerate(L):
        ins.append(t)
        s = t @ W[:, 1:].T
        s[0] += W[:, 0]
        if l < len(L) - 1:
            t, u = se.tanh(s)
            us.append(u)
    return L, ins, us, (s[:, :, 0] * se.fact.view(-1, 1)).T


def _backward(se, L, ins, us, seed, rows=False):
    """dL/dw from seed[P][na] = dL/dT, summed over the points or per point."""
    sb = (seed.T * se.fact.view(-1, 1)).unsqueeze(2)
    out = [None] * len(L)
    for l in range(len(L) - 1, -1, -1):
        if rows:
            g = torch.einsum("apn,apm->pnm", sb, ins[l])
            out[l] = torch.cat([sb[0].unsqueeze(2), g], 2).reshape(sb.shape[1], -1)
        else:
            g = torch.einsum("apn,apm->nm", sb, ins[l])
            out[l] = torch.cat([sb[0].sum(0).unsqueeze(1), g], 1).reshape(-1)
        if l:
            sb = se.adjoint(sb @ L[l][:, 1:], us[l - 1])
    return torch.cat(out, 1 if rows else 0)


def _residual(terms, T):
    R = torch.zeros(T.shape[0], dtype=T.dtype, device=T.device)
    dR = torch.zeros_like(T)
    for co, slot, nl in terms:
        v = T[:, slot - 1]
        R = R + co * (T[:, 0] * v if nl else v)
        if nl:
            dR[:, slot - 1] += co * T[:, 0]
            dR[:, 0] += co * v
        else:
            dR[:, slot - 1] += co
    return R, dR


def _chunks(se, c, x):
    per = 8 * 3 * len(se.pairs[0]) * c["width"]
    n = max(1, int(16e9 // per))
    return x.split(n)


def _sweep(c, w, x, terms, rows=False, halfsq=False):
    se = _Series(c, x.device)
    loss, g, res, rw = 0.0, 0.0, [], []
    for xc in _chunks(se, c, x):
        L, ins, us, T = _forward(se, c, w, xc)
        if halfsq:
            loss, seed = loss + 0.5 * (T * T).sum(), T
        else:
            R, dR = _residual(terms, T)
            loss, seed = loss + 0.5 * (R * R).sum(), R.unsqueeze(1) * dR
            res.append(R)
        g = g + _backward(se, L, ins, us, seed)
        if rows:
            rw.append(_backward(se, L, ins, us, dR, rows=True))
    return loss, g, torch.cat(res) if res else None, torch.cat(rw) if rw else None


def _update(P, w, j, xi, lam):
    """One rank-one filter update (weights, covariance, lambda)."""
    p = P @ j
    den = lam + j @ p
    kv = p / den
    w += kv * xi
    P -= torch.outer(kv, p)
    P /= lam
    return KF[2] * lam + 1.0 - KF[2]


def exact(case, seed):
    c = dict(case)
    r = np.random.default_rng(seed)
    dev = DEV if torch.cuda.is_available() else "cpu:0"
    if c["kind"] == "committee":
        loss, grads = [], []
        for m in _members(c):
            w = torch.tensor(_weights(_dims(m), r), device=dev)
            x = torch.tensor(_points(m, r), device=dev)
            lo, g, _, _ = _sweep(m, w, x, None, halfsq=True)
            loss.append(lo)
            grads.append(g)
        return {"loss": torch.stack(loss), "grads": grads}
    w = torch.tensor(_weights(_dims(c), r), device=dev)
    nw = w.numel()
    if c["kind"] == "kf_rows":
        rows, xi = _rows(c, nw, seed)
        P = torch.eye(nw, dtype=torch.float64, device=dev) * KF[0]
        lam = KF[1]
        for k in range(c["npts"]):
            lam = _update(P, w, rows[k], xi[k], lam)
        return {"w": w}
    x = torch.tensor(_points(c, r), device=dev)
    alpha = _alpha(c)
    if c["kind"] == "eval":
        se = _Series(c, x.device)
        T = torch.cat([_forward(se, c, w, xc)[3] for xc in _chunks(se, c, x)])
        return T[0] if c["npts"] == 1 else T
    terms = _terms(c, alpha)
    if c["kind"] == "kf_pass":
        P = torch.eye(nw, dtype=torch.float64, device=dev) * KF[0]
        lam = KF[1]
        se = _Series(c, x.device)
        for k in range(c["npts"]):
            L, ins, us, T = _forward(se, c, w, x[k:k + 1])
            R, dR = _residual(terms, T)
            j = _backward(se, L, ins, us, dR)
            lam = _update(P, w, j, -R[0], lam)
        return {"w": w, "lam": torch.tensor(lam, dtype=torch.float64)}
    if c["kind"] == "epoch":
        loss, g, _, _ = _sweep(c, w, x, terms, halfsq=c["k"] <= 3)
        eta, b1, b2, eps = ADAM
        gv = g / c["npts"]
        m, v = (1.0 - b1) * gv, (1.0 - b2) * gv * gv
        return {"loss": loss, "grad": g,
                "w": w - eta * (m / (1.0 - b1)) / (torch.sqrt(v / (1.0 - b2)) + eps)}
    if c["kind"] == "autograd" and c["prec"]:
        w = w.float().double()           # the parameters the program holds
    loss, g, res, rows = _sweep(c, w, x, terms, rows=c["kind"] == "ngd")
    if c["kind"] == "autograd":
        return {"loss": loss, "grad": g, "res": res}
    if c["kind"] == "colloc":
        return {"loss": loss.view(1), "grad": g}
    G = rows.T @ rows / c["npts"]
    G.diagonal().add_(c["mu"])
    u = torch.linalg.solve(G, g / c["npts"])
    return {"u": u, "grad": g, "loss": loss.view(1)}
