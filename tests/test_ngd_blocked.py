"""The blocked FP64 Cholesky solve and the FP64 metric product at the edges
of their 64-wide panels and tiles, against numpy.

Bounds: a product of n terms is within (n + 2) eps of the sum of its terms'
magnitudes (in the split precision with the unit roundoff of FP32), and the solve's backward error within 3 n eps (the factor and the
two substitutions, each n eps)."""
import numpy as np
import pytest

from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
SIZES = [1, 2, 63, 64, 65, 127, 128, 129, 200, 448, 641]


def _dev(a):
    import torch
    return torch.tensor(a, device="cuda")


def _gram(J, prec=0):
    import torch
    nrow, nw = J.shape
    Jd = _dev(J)
    G = torch.full((nw, nw), float("nan"), dtype=torch.float64, device="cuda")
    api.call("dnnf90_ngd_gram_dev", nrow, nw, Jd.data_ptr(), prec, G.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    return G


@pytest.mark.parametrize("nw", SIZES)
@pytest.mark.parametrize("nrow", [1, 15, 16, 17, 300, 1100])
@pytest.mark.parametrize("prec", [0, 1])
def test_metric(nw, nrow, prec):
    J = np.random.default_rng(nw + nrow).normal(size=(nrow, nw))
    G = np.tril(_gram(J, prec).cpu().numpy())
    # split: an FP32 copy (2 u), the dropped terms of order 3 (4 u), and FP32
    # sums of six products over runs of at most 512 rows, u = 2^-24
    terms = (nrow + 2) * EPS if prec == 0 else (6 + 6 * min(nrow, 512)) * 2.0 ** -24
    bound = terms * (np.abs(J).T @ np.abs(J))
    assert np.all(np.abs(G - np.tril(J.T @ J)) <= np.tril(bound) + 1e-300)


@pytest.mark.parametrize("n", SIZES)
def test_solve(n):
    import torch
    rng = np.random.default_rng(n)
    J = rng.normal(size=(n // 2 + 1, n))
    nb, mu = n // 2 + 1, 1e-2
    A = J.T @ J / nb + mu * np.eye(n)
    b = rng.normal(size=n)
    G = torch.tril(_dev(J.T @ J)).contiguous()
    u = torch.empty(n, dtype=torch.float64, device="cuda")
    bd = _dev(b)
    api.call("dnnf90_ngd_solve_dev", n, G.data_ptr(), bd.data_ptr(), nb, mu, u.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    x = u.cpu().numpy()
    an = np.linalg.norm(A, 2)
    berr = np.linalg.norm(A @ x - b / nb) / (an * np.linalg.norm(x) + np.linalg.norm(b / nb))
    assert berr <= 3 * n * EPS, berr
    L = np.tril(G.cpu().numpy())
    assert np.linalg.norm(L @ L.T - A) <= 3 * n * EPS * np.linalg.norm(A) * np.sqrt(n)
    assert np.all(np.triu(G.cpu().numpy(), 1) == 0.0)


@pytest.mark.parametrize("n,bad", [(40, 7), (130, 64), (130, 65), (200, 199)])
def test_indefinite_is_refused(n, bad):
    """The first non-positive pivot is named (1-based) and the call fails."""
    import torch
    G = torch.eye(n, dtype=torch.float64, device="cuda") * 2.0
    G[bad - 1, bad - 1] = -1.0
    G[n - 1, n - 1] = -1.0
    b, u = torch.ones(n, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    rc = api.lib().dnnf90_ngd_solve_dev(n, G.data_ptr(), b.data_ptr(), 1, 0.0, u.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
    assert rc == -1 and f"column {min(bad, n)}".encode() in api.lib().dnnf90_last_error()


@pytest.mark.parametrize("nrow,nw", [(1, 5), (64, 65), (65, 300), (190, 131)])
def test_dual(nrow, nw):
    import torch
    rng = np.random.default_rng(nrow)
    J, b, mu = rng.normal(size=(nrow, nw)), rng.normal(size=nw), 1e-1
    Jd, bd = _dev(J), _dev(b)
    u = torch.full((nw,), float("nan"), dtype=torch.float64, device="cuda")
    api.call("dnnf90_ngd_step_dual_dev", nrow, nw, Jd.data_ptr(), bd.data_ptr(), nrow, mu,
             u.data_ptr(), torch.cuda.current_stream().cuda_stream)
    A = J.T @ J / nrow + mu * np.eye(nw)
    ref = np.linalg.solve(A, b / nrow)
    cond = np.linalg.cond(A)
    assert np.linalg.norm(u.cpu().numpy() - ref) <= 10 * (nrow + nw) * EPS * cond * np.linalg.norm(ref)
