"""The natural-gradient step written over its own right-hand side, by every
route, against the same step into another array (equal bits: nothing but the
destination differs), and against numpy within the solve's backward error (see
test_ngd_blocked.py); and the dual step's bits from call to call."""
import numpy as np
import pytest

from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


def _problem(nrow, nw):
    import torch
    rng = np.random.default_rng(nrow + nw)
    J, b = rng.normal(size=(nrow, nw)), rng.normal(size=nw)
    return J, b, torch.tensor(J, device="cuda"), torch.tensor(b, device="cuda")


def _step(route, Jd, b, u, mu):
    import torch
    nrow, nw = Jd.shape
    st = torch.cuda.current_stream().cuda_stream
    if route == "dual":
        api.call("dnnf90_ngd_step_dual_dev", nrow, nw, Jd.data_ptr(), b.data_ptr(), nrow, mu,
                 u.data_ptr(), st)
    elif route == "noalloc":
        api.call("dnnf90_ngd_step_noalloc", nrow, nw, Jd.data_ptr(), b.data_ptr(), nrow, mu,
                 u.data_ptr(), st)
    else:
        G = torch.empty((nw, nw), dtype=torch.float64, device="cuda")
        api.call("dnnf90_ngd_gram_dev", nrow, nw, Jd.data_ptr(), 0, G.data_ptr(), st)
        api.call("dnnf90_ngd_solve_dev", nw, G.data_ptr(), b.data_ptr(), nrow, mu, u.data_ptr(),
                 st)
    torch.cuda.synchronize()


@pytest.mark.parametrize("nrow,nw", [(1, 5), (16, 129), (17, 64), (100, 300), (300, 60)])
@pytest.mark.parametrize("route", ["dual", "primal", "noalloc"])
def test_step_in_place(route, nrow, nw):
    import torch
    J, b, Jd, bd = _problem(nrow, nw)
    mu = 1e-2
    u = torch.full_like(bd, float("nan"))
    _step(route, Jd, bd, u, mu)
    assert np.array_equal(bd.cpu().numpy(), b)  # the right-hand side is read only
    x = bd.clone()
    _step(route, Jd, x, x, mu)
    if (nw if route == "dual" else nrow) <= 64:  # a metric of one slab: no order of additions
        assert np.array_equal(x.cpu().numpy(), u.cpu().numpy())
    A = J.T @ J / nrow + mu * np.eye(nw)
    uref = np.linalg.solve(A, b / nrow)
    # the dual route divides a difference by mu, which costs the condition twice
    cond = np.linalg.cond(A) ** (2 if route == "dual" else 1)
    err = np.linalg.norm(x.cpu().numpy() - uref) / np.linalg.norm(uref)
    assert err <= 3 * (nrow + nw) * 2.0 ** -52 * cond


def test_dual_step_repeats_its_bits():
    import torch
    _, _, Jd, bd = _problem(300, 60)
    out = []
    for _ in range(4):
        u = torch.empty_like(bd)
        _step("dual", Jd, bd, u, 1e-3)
        out.append(u.cpu().numpy())
    assert all(np.array_equal(out[0], o) for o in out[1:])
