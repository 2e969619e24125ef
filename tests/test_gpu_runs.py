"""The run kernels (9 gathered rows per slot, y taps as shifted reads) against the kernels that gather every tap by itself, at the
edges of their tile shapes.  The forward pass keeps the order of the products: equal bit for bit.  The input gradient may add the
same products in another order: relative difference (2-norm) at most 2e-6, a few fp32 roundings of sums of unit scale.  The same
bound holds for the weight gradient, whose sums run over all locations."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu

WIDTHS = [(8, 8), (16, 40), (33, 33), (32, 32), (64, 32), (32, 64), (96, 64), (24, 120), (64, 128), (128, 128), (48, 17), (130, 32)]


def _run(apr, dl, cin, cout, n):
    from pyapr.aprnet import cuda as ops
    torch.manual_seed(1)
    conv = ops.APRConv(cin, cout, nstencils=2, precision="bf16").cuda()
    x = torch.randn(1, cin, n, device="cuda").requires_grad_(True)
    g = torch.randn(1, cout, n, device="cuda")
    out = conv(x, [apr], torch.full((1,), dl, dtype=torch.int32))
    out.backward(g)
    return out.detach(), x.grad, conv.weight.grad


@pytest.mark.parametrize("name", ["blob", "odd", "plane", "ref_shape"])
@pytest.mark.parametrize("cin,cout", WIDTHS)
def test_run_kernels_match_the_tap_kernels(name, cin, cout):
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    a = H.arrays(name) if name in H.APR_CASES else H.blob_arrays()
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    for dl in range(0, H.max_dl(a) + 1):
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        try:
            C.tc_set_option("runs", 0)
            want = _run(apr, dl, cin, cout, n)
        finally:
            C.tc_set_option("runs", 1)
        got = _run(apr, dl, cin, cout, n)
        assert C.tc_error_flag() == 0
        assert torch.equal(got[0], want[0]), (dl, int((got[0] != want[0]).sum()))
        for k in (1, 2):
            assert float((got[k] - want[k]).norm() / want[k].norm()) <= 2e-6, (dl, k)
