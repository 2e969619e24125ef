"""Rounding of the 3x3x3 weight gradient against float64 on the same operands: 2 M locations, so that sums are long.

fp32: products are added in chains of L = max(512, 1 / 256 of the level) locations at most.  The partial sums of terms of random sign
grow like sqrt(k), each addition rounds to 2^-24 of them (0.41 of that, rms): relative 2-norm 0.29 * sqrt(L) * 2^-24.

bf16 operands (exact here, the tree means as they are rounded): the tensor cores truncate, so the error grows with the D products of
16 locations that an accumulator takes one after the other: 0.3 * D * 2^-24, with D as two waves of blocks leave that fill TMEM."""
import math

import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,dl", [(16, 16, 0), (33, 33, 0), (32, 64, 0), (64, 64, 0), (128, 128, 1)])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_weight_gradient_rounding(cin, cout, dl, precision):
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.blob_arrays((128, 256, 256), 800, 5)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    v = APRPtrVector([apr])
    n = int(pyapr.aprnet.utils.number_particles(apr, dl))
    ld = torch.full((1,), dl, dtype=torch.int32)
    torch.manual_seed(1)
    x = torch.randn(1, cin, n, device="cuda").relu_()
    g = torch.randn(1, cout, n, device="cuda")
    if precision == "bf16":
        x, g = x.bfloat16().float(), g.bfloat16().float()
    w = torch.randn(a.level_max - a.level_min + 1, cout, cin, 3, 3, 3, device="cuda") / (27 * cin) ** 0.5
    _, rows = C.conv333_forward_keep_rows(v, x, w, ld, precision)
    got = [C.conv333_backward_with_rows(v, rows, w, g, ld, False, precision)[1] for _ in range(2)]
    assert torch.equal(got[0], got[1])
    tree = C.conv333_forward_keep_tree(v, x, w, ld, "fp32")[1]
    if precision == "bf16":
        tree = tree.bfloat16()
    want = C.conv333_backward_pretree(v, x.double(), tree.double(), torch.empty(0, dtype=torch.uint8, device="cuda"), w.double(),
                                      g.double(), ld, False)[2]
    if precision == "fp32":
        bound = 0.29 * math.sqrt(max(512, n / 256)) * 2.0 ** -24
    else:
        full = math.ceil(27 * ((cin + 15) // 16 * 16) * ((cout + 63) // 64 * 64) / 65536)
        bound = 0.3 * 8 * math.ceil(n / 128 * full / (2 * 148)) * 2.0 ** -24
    assert float((got[0] - want).norm() / want.norm()) <= bound
