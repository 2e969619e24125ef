"""The run kernels (9 gathered rows per slot, y taps as shifted reads) at the edges of their tile shapes.

Forward pass and input gradient against the kernels that gather every tap by itself (`runs` = 0).  The forward pass keeps the order
of the products: equal bit for bit (from 128 channels on each side both arms are the tap kernel).  The input gradient may add
the same products in another order: relative difference (2-norm) at most 2e-6, a few fp32 roundings of sums of unit scale.

The weight gradient always runs over the slots; it is held against the float64 kernel on the same operands: features and gradients
that are exact in bf16, and the tree means as they are rounded to bf16.  What is left is the rounding of fp32 sums: the tensor cores truncate, so an accumulator that takes DEPTH products of 16 slots one after the
other loses at most DEPTH * 2^-23 of sums of its own size."""
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
        assert float((got[1] - want[1]).norm() / want[1].norm()) <= 2e-6, dl


@pytest.mark.parametrize("cin,cout", [(16, 128), (40, 72), (48, 128), (96, 128), (160, 100), (33, 20), (48, 64), (128, 48)])
def test_run_kernels_of_padded_and_wide_layers(cin, cout):
    """Stages of 48 channels, and forward layers of 65 to 128 result channels whose stages of the tap kernel hold three taps; several tiles per block."""
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    apr = pyapr.apr_from_arrays(H.blob_arrays((64, 128, 128), 40, 11))
    apr.init_cuda()
    for dl in (0, 1):
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        try:
            C.tc_set_option("runs", 0)
            want = _run(apr, dl, cin, cout, n)
        finally:
            C.tc_set_option("runs", 1)
        got = _run(apr, dl, cin, cout, n)
        assert C.tc_error_flag() == 0
        assert torch.equal(got[0], want[0]), (dl, int((got[0] != want[0]).sum()))
        assert float((got[1] - want[1]).norm() / want[1].norm()) <= 2e-6, dl


@pytest.mark.parametrize("cin,cout", [(128, 128), (113, 65), (192, 100), (256, 128), (320, 72), (448, 128), (1024, 70)])
@pytest.mark.parametrize("name", ["odd", "volume", "large"])
def test_wide_forward_layers_keep_their_order(name, cin, cout):
    """Forward layers whose taps run one after the other over all source channels: tiles of one and two blocks of rows, up to
    the widths whose rows no longer fit, and structures that stay with the tap kernel; bit for bit what the kernel that gathers every tap gives."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    a = H.arrays(name) if name == "odd" else H.blob_arrays((64, 128, 128), 40, 11) if name == "volume" else H.blob_arrays((128, 128, 160), 200, 3)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(2)
    conv = ops.APRConv(cin, cout, nstencils=3, precision="bf16").cuda()
    for dl in (0, 1): 
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        x, ld = torch.randn(1, cin, n, device="cuda"), torch.full((1,), dl, dtype=torch.int32)
        with torch.no_grad():
            try:
                C.tc_set_option("runs", 0)
                want = conv(x, [apr], ld)
            finally:
                C.tc_set_option("runs", 1)
            got = conv(x, [apr], ld)
        assert C.tc_error_flag() == 0
        assert torch.equal(got, want), (dl, int((got != want).sum()))


# widths with one stage per chunk of slots (more than 64 output channels, the last neighbour group of wide inputs) and with several
DW_WIDTHS = [(8, 8), (16, 40), (33, 33), (64, 32), (24, 120), (32, 128), (128, 64), (128, 128), (130, 32), (48, 200)]


@pytest.mark.parametrize("name", ["blob", "odd", "plane", "many_chunks"])
@pytest.mark.parametrize("cin,cout", DW_WIDTHS)
def test_weight_gradient_matches_float64(name, cin, cout):
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    if name == "many_chunks":              # hundreds of chunks per block: the dO buffers and the ring go round many times
        a = H.blob_arrays((128, 128, 128), 200, 12)
    else:
        a = H.arrays(name) if name in H.APR_CASES else H.blob_arrays()
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    L = a.level_max - a.level_min + 1
    for dl in (0,) if name == "many_chunks" else range(0, H.max_dl(a) + 1):
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        ld = torch.full((1,), dl, dtype=torch.int32)
        torch.manual_seed(2)
        x = torch.randn(1, cin, n, device="cuda").bfloat16().float()
        g = torch.randn(1, cout, n, device="cuda").bfloat16().float()
        w = torch.randn(L, cout, cin, 3, 3, 3, device="cuda") / (27 * cin) ** 0.5
        v = APRPtrVector([apr])
        _, rows = C.conv333_forward_keep_rows(v, x, w, ld, "bf16")
        runs = [C.conv333_backward_with_rows(v, rows, w, g, ld, False, "bf16")[1] for _ in range(3)]
        assert C.tc_error_flag() == 0
        assert all(torch.equal(r, runs[0]) for r in runs[1:])          # one order of summation
        tree = C.conv333_forward_keep_tree(v, x, w, ld, "fp32")[1]
        if cin > 4: tree = tree.bfloat16()
        want = C.conv333_backward_pretree(v, x.double(), tree.double(), torch.empty(0, dtype=torch.uint8, device="cuda"), w.double(),
                                          g.double(), ld, False)[2]
        depth = 1.27 * n / 16          # all slots in one accumulator: more than any block takes
        assert float((runs[0] - want).norm() / want.norm()) <= depth * 2.0 ** -23, (dl, float((runs[0] - want).norm() / want.norm()))
