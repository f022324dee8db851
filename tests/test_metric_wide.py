"""The split metric of a network with more tiles in its triangle than one
grid dimension holds (65535 of 128 x 128: beyond 46208 weights): the
tensor-core route, at the tiles on both sides of that count.  Bound of a
product as in test_ngd_blocked.py."""
import numpy as np
import pytest

from dnnf90_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [46208, 46209, 46500])
def test_split_metric_beyond_one_grid_dimension(nw):
    import torch
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 17 GiB for the metric")
    nrow = 40
    torch.manual_seed(nw)
    J = torch.randn((nrow, nw), dtype=torch.float64, device="cuda")
    G = torch.empty((nw, nw), dtype=torch.float64, device="cuda")
    api.profile_enable(True)
    api.profile_read()
    api.call("dnnf90_ngd_gram_dev", nrow, nw, J.data_ptr(), api.PREC_SPLIT, G.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    names = api.profile_read()
    api.profile_enable(False)
    assert "k_tc_syrk" in names and "k_syrk_f64" not in names, names
    bound = (6 + 6 * nrow) * 2.0 ** -24
    # whole rows: the first, some inside, and all of the last tiles'
    rows = [0, 127, 128, 20000, 46000] + list(range(nw - 130, nw))
    for r in rows:
        want = J[:, r] @ J[:, :r + 1]
        mag = J[:, r].abs() @ J[:, :r + 1].abs()
        assert bool(torch.all((G[r, :r + 1] - want).abs() <= bound * mag + 1e-300)), r
    del J, G
    torch.cuda.empty_cache()
