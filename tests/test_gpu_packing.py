"""Packed bf16 rows of the features: any number of channels, and none of them on a slower path than a wider layer."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


def _apr(arrays):
    import pyapr
    apr = pyapr.apr_from_arrays(arrays)
    apr.init_cuda()
    return apr


@pytest.mark.parametrize("c", [5, 8, 16, 17, 24, 31, 33, 48, 65])
@pytest.mark.parametrize("name", ["odd", "volume"])
def test_rows_of_any_width(name, c):
    """A row holds the rounded channels of its location and zeros behind them."""
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.blob_arrays((64, 128, 128), 40, 11) if name == "volume" else H.arrays(name)
    apr = _apr(a)          # (the vector of pointers does not keep it)
    torch.manual_seed(c)
    x = torch.randn(1, c, a.n_particles, device="cuda")
    w = torch.zeros(a.level_max - a.level_min + 1, 8, c, 3, 3, 3, device="cuda")
    rows = C.conv333_forward_keep_rows(APRPtrVector([apr]), x, w, torch.zeros(1, dtype=torch.int32), "bf16")[1]
    pad = (c + 15) // 16 * 16
    got = rows.view(torch.bfloat16).flatten()[:a.n_particles * pad].view(a.n_particles, pad)
    assert torch.equal(got[:, :c], x[0].t().bfloat16()) and bool((got[:, c:] == 0).all())


@pytest.mark.parametrize("narrow,wide", [(8, 32), (16, 32), (24, 64), (48, 64)])
def test_narrow_rows_are_not_slower_than_wide_ones(narrow, wide):
    """Both are bound by the bytes they move, of which the narrow ones have at most 3/4."""
    import pyapr
    from pyapr import synthetic
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    apr = _apr(synthetic.apr_from_level_map(torch.full((64, 64, 64), 7, dtype=torch.int16), (128, 128, 128)))
    n, took = int(pyapr.aprnet.utils.number_particles(apr, 0)), {}
    with torch.no_grad():
        for c in (narrow, wide):
            conv, x, ld = ops.APRConv(c, 8, precision="bf16").cuda(), torch.randn(1, c, n, device="cuda"), torch.zeros(1, dtype=torch.int32)
            best = []
            for _ in range(7):
                conv(x, [apr], ld)
                torch.cuda.synchronize()
                C.profile_enable(True)
                try:
                    conv(x, [apr], ld)
                    torch.cuda.synchronize()
                    best.append(C.profile_read()["pack_rows_bf16"][1])
                finally:
                    C.profile_enable(False)
            took[c] = min(best)
    assert took[narrow] < took[wide], took
