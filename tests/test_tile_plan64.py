"""The FP64 register-tiled Bell kernels: their work lists on the CPU
(tests/cpp/tile_plan64_check.cpp, every dense set with D0 <= 4 and K <= 7),
and the kernels, pinned, against the oracle on the GPU at 1e-12: ragged
16-neuron tiles, one point, K from 1 to 7, D0 from 1 to 5."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import pyoracle as po
from conftest import ROOT, per_order_error, rel_err, xavier_weights
from dnnf90_b200 import api


def test_work_lists(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no C++ compiler")
    csrc = os.path.join(ROOT, "dnnf90_b200", "csrc")
    exe = str(tmp_path / "tile_plan64_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", csrc,
                    os.path.join(ROOT, "tests", "cpp", "tile_plan64_check.cpp"),
                    os.path.join(csrc, "tile_plan.cpp"), os.path.join(csrc, "tables.cpp"),
                    "-o", exe], check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and "ALL OK" in out.stdout, out.stdout[-3000:]


@pytest.mark.gpu
@pytest.mark.parametrize("d0,k,dims,npts", [
    (4, 7, [4, 64, 18, 1], 5), (4, 7, [4, 16, 16, 1], 1), (4, 5, [4, 30, 46, 1], 40),
    (3, 7, [3, 100, 44, 1], 9), (3, 2, [3, 10, 6, 1], 300), (2, 7, [2, 34, 34, 1], 33),
    (1, 3, [1, 16, 20, 1], 7), (4, 1, [4, 32, 32, 1], 20), (5, 4, [5, 20, 20, 1], 3)])
@pytest.mark.parametrize("act", [0, 1])
def test_pinned_against_the_oracle(d0, k, dims, npts, act):
    ts, ref = api.TableSet(d0, k, activation=act), po.Tables(d0, k, activation=act)
    w = xavier_weights(dims, 23)
    w[np.arange(len(w)) % 6 == 0] += 0.04
    X = np.random.default_rng(4).uniform(-1, 1, (npts, d0))
    net = api.Net(ts, dims, weights=w)
    g, r = net.grad(), api.SeedRule(api.SEED_HALFSQ)
    try:
        api.tune_force(0, 3)
        api.tune_force(1, 3)
        loss, T = g.rule_batch(X, r, want_t=True)
        Te = net.eval(X if npts > 1 else X[0])
    finally:
        api.tune_force(0, -1)
        api.tune_force(1, -1)
    gref, Tref, lref, _ = po.grad_batch(ref, dims, w, X)
    assert max(per_order_error(T, Tref, ref.deg).values()) < 1e-12
    assert np.array_equal(Te.reshape(T.shape), T)
    assert rel_err(g.read(), gref) < 1e-12 and abs(loss - lref) <= 1e-12 * abs(lref)
    r.free(); g.free(); net.free(); ts.free()
