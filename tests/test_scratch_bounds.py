"""Device memory that calls take for themselves: after a call with large scratch
the device has all but a bounded part of it back, without a further call."""
import pytest

from dnnf90_b200 import api

pytestmark = pytest.mark.gpu
KEEP = 512 << 20


def _used():
    import torch
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("route", ["split_metric", "dual"])
def test_large_scratch_goes_back(route):
    import torch
    nrow, nw = (30000, 12000) if route == "split_metric" else (9000, 30000)
    J = torch.randn((nrow, nw), dtype=torch.float64, device="cuda")
    G = torch.empty((nw, nw), dtype=torch.float64, device="cuda") if route == "split_metric" else None
    b = torch.randn(nw, dtype=torch.float64, device="cuda")
    u = torch.empty_like(b)
    st = torch.cuda.current_stream().cuda_stream

    def run(n):
        if route == "split_metric":  # an FP32 copy of the rows: 1.4 GB
            api.call("dnnf90_ngd_gram_dev", n, nw, J.data_ptr(), api.PREC_SPLIT, G.data_ptr(), st)
        else:                        # the rows transposed and their Gram matrix: 2.8 GB
            api.call("dnnf90_ngd_step_dual_dev", n, nw, J.data_ptr(), b.data_ptr(), n, 1e-2,
                     u.data_ptr(), st)

    run(64)                          # loads the kernels
    torch.cuda.synchronize()
    base = _used()
    run(nrow)
    assert _used() - base <= KEEP + (64 << 20)
    run(nrow)
    assert _used() - base <= KEEP + (64 << 20)
    del J, G, b, u
    torch.cuda.empty_cache()
