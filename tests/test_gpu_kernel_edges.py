"""Sizes at which the copies of pooling, the GroupNorm kernels, the sums of the cross-level part and the wide forward layers change their shape; sums of
subnormal values."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


def _apr(a):
    import pyapr
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    return apr


# rows of one tile and less, of a tile and one more, of many tiles per block; every alignment of a row comes up where n is odd
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("c,n", [(3, 1), (5, 31), (3, 993), (7, 1024), (4, 2049), (1, 300001)])
def test_groupnorm_row_lengths(c, n, dtype):
    from pyapr.aprnet import cuda as ops
    torch.manual_seed(4)
    x = torch.randn(2, c, n, dtype=dtype, device="cuda").requires_grad_(True)
    m = ops.GroupNormReLU(1, c).to("cuda", dtype)
    g = torch.randn_like(x)
    y = m(x)
    y.backward(g)
    xd = x.detach().double().requires_grad_(True)
    want = torch.relu(torch.nn.functional.group_norm(xd, 1, eps=1e-5))
    # the ReLU's gate is taken from the computed output: a value within rounding of zero has either
    want.backward(torch.where((y > 0) == (want > 0), g, torch.zeros_like(g)).double())
    eps = 2.0 ** -23 if dtype == torch.float32 else 2.0 ** -52
    assert float((y - want).abs().max()) <= 8 * eps * float(want.abs().max())
    same = (y > 0) == (want > 0)
    assert float((~same).sum()) <= 1e-4 * n * c + 1
    if bool(same.all()):
        assert float((x.grad - xd.grad).norm()) <= 64 * eps * float(xd.grad.norm()) + 1e-30


def _two_levels(refined):
    """5 x 10 x 41 cells of one level, the first few of every 700 divided once: 2050 - refined particles below the finest level."""
    from pyapr import synthetic
    level_map = torch.full((5, 10, 41), 6, dtype=torch.int32)
    level_map.view(-1)[torch.arange(refined) * 700] = 7
    return synthetic.apr_from_level_map(level_map, (10, 20, 82))


# the copy kernel's blocks take 2048 entries each, shifted by where a row starts in its 128-byte line: one entry less, as many, one more, and
# several blocks with a ragged end.  Five channels of rows of odd length start at five places of a line
@pytest.mark.parametrize("refined,count", [(3, 2047), (2, 2048), (1, 2049), (None, None)])
@pytest.mark.parametrize("channels", [1, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_pooling_keeps_coarse_particles(refined, count, channels, dtype):
    """The particles below the finest level come through pooling and up-sampling bit for bit."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays((64, 96, 112), 40, 8) if refined is None else _two_levels(refined)
    kept = int(a.row_ptr[sum(a.dims[l][0] * a.dims[l][1] for l in range(a.level_min, a.level_max))])
    assert kept == count if count else kept > 4096
    apr = _apr(a)
    for pad in (1, 2):
        x = torch.randn(1, channels, a.n_particles + pad, dtype=dtype, device="cuda")
        ld = torch.zeros(1, dtype=torch.int32)
        pooled = ops.MaxPool()(x, [apr], ld)
        assert pooled.shape[2] == int(pyapr.aprnet.utils.number_particles(apr, 1))
        up = ops.UpSampleConst()(pooled, [apr], ld)
        assert torch.equal(pooled[..., :kept], x[..., :kept]) and torch.equal(up[..., :kept], x[..., :kept])


@pytest.mark.parametrize("cin,cout", [(16, 40), (16, 272), (24, 520)])
def test_cross_level_sums_of_ragged_widths(cin, cout):
    """Row widths that do not divide a block's threads and that take several columns of blocks, against the float64 kernels on operands that are exact in
    bf16: what is left is the rounding of the sums (to bf16, 2^-9) and of the tree means."""
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.blob_arrays((48, 64, 64), 8, 5)
    apr = _apr(a)
    L = a.level_max - a.level_min + 1
    n = int(pyapr.aprnet.utils.number_particles(apr, 0))
    ld = torch.zeros(1, dtype=torch.int32)
    torch.manual_seed(5)
    w = (torch.randn(L, cout, cin, 3, 3, 3, device="cuda") / (27 * cout) ** 0.5).bfloat16().float()
    g = torch.randn(1, cout, n, device="cuda").bfloat16().float()
    x = torch.randn(1, cin, n, device="cuda")
    v = APRPtrVector([apr])
    _, rows = C.conv333_forward_keep_rows(v, x, w, ld, "bf16")
    got = C.conv333_backward_with_rows(v, rows, w, g, ld, True, "bf16")[0]
    want = C.conv333_backward(v, x.double(), w.double(), g.double(), ld)[0]
    assert C.tc_error_flag() == 0
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -9


@pytest.mark.parametrize("cin,cout", [(16, 16), (33, 40), (72, 17), (130, 24)])
@pytest.mark.parametrize("dl", [0, 1])
def test_cross_level_sums_keep_subnormal_values(cin, cout, dl):
    """Gradients below the smallest normal number: the operands are small whole numbers times powers of two, so every product, sum and tree
    adjoint (factors 1/8 to 1) is exact, and scaling the operands scales the input gradient bit for bit down to 2^-149."""
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.arrays("odd")
    apr = _apr(a)
    n = int(pyapr.aprnet.utils.number_particles(apr, dl))
    ld = torch.full((1,), dl, dtype=torch.int32)
    torch.manual_seed(1)
    w = torch.randint(-2, 3, (a.level_max - a.level_min + 1, cout, cin, 3, 3, 3), device="cuda").float()
    g = torch.randint(-3, 4, (1, cout, n), device="cuda").float()
    v, x = APRPtrVector([apr]), torch.zeros(1, cin, n, device="cuda")
    _, rows = C.conv333_forward_keep_rows(v, x, w, ld, "bf16")
    plain = C.conv333_backward_with_rows(v, rows, w, g, ld, True, "bf16")[0].double()
    assert torch.equal(plain, C.conv333_backward(v, x.double(), w.double(), g.double(), ld)[0])
    want = plain * 2.0 ** -133
    assert int(((want != 0) & (want.abs() < 2.0 ** -126)).sum()) > n and bool((want * 2.0 ** 149 == (want * 2.0 ** 149).round()).all())
    got = C.conv333_backward_with_rows(v, rows, w * 2.0 ** -66, g * 2.0 ** -67, ld, True, "bf16")[0].double()
    assert C.tc_error_flag() == 0 and torch.equal(got, want)


# narrow result tiles on few tiles of locations, one and two blocks of 128 slots per tile on many
STRUCTURES = [("odd",), ((64, 96, 96), 30, 6), ((128, 128, 256), 200, 6)]


@pytest.mark.parametrize("cin,cout", [(16, 65), (16, 128), (32, 100), (64, 127), (64, 128)])
@pytest.mark.parametrize("structure", STRUCTURES)
def test_wide_forward_layers_over_runs(cin, cout, structure):
    """65 to 128 result channels with all source channels in one stage: over runs of cells (`runs` = 1) the same bits as tap by tap (0)."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    apr = _apr(H.blob_arrays(*structure) if len(structure) > 1 else H.arrays(*structure))
    n = int(pyapr.aprnet.utils.number_particles(apr, 0))
    torch.manual_seed(6)
    conv = ops.APRConv(cin, cout, nstencils=2, precision="bf16").cuda()
    x = torch.randn(1, cin, n, device="cuda")
    ld = torch.zeros(1, dtype=torch.int32)
    out = {}
    with torch.no_grad():
        for runs in (0, 1):
            C.tc_set_option("runs", runs)
            try:
                out[runs] = conv(x, [apr], ld)
            finally:
                C.tc_set_option("runs", 1)
    assert C.tc_error_flag() == 0 and torch.equal(out[0], out[1])


@pytest.mark.parametrize("cin,cout", [(16, 130), (48, 256), (64, 200), (160, 264), (128, 128)])
@pytest.mark.parametrize("structure", STRUCTURES[:2])
def test_wide_forward_layers_tap_by_tap(cin, cout, structure):
    """Wider layers, against the float64 kernel on operands that are exact in bf16 (features, stencils, tree means as they are rounded): an accumulator takes
    27 products of 16 channels per block of them, one after the other, and the tensor cores truncate each sum by at most 2^-23 of its size.  A
    bias is one addition more."""
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.blob_arrays(*structure) if len(structure) > 1 else H.arrays(*structure)
    apr = _apr(a)
    n = int(pyapr.aprnet.utils.number_particles(apr, 0))
    ld = torch.zeros(1, dtype=torch.int32)
    torch.manual_seed(7)
    w = (torch.randn(a.level_max - a.level_min + 1, cout, cin, 3, 3, 3, device="cuda") / (27 * cin) ** 0.5).bfloat16().float()
    x = torch.randn(1, cin, n, device="cuda").bfloat16().float()
    v = APRPtrVector([apr])
    got, _ = C.conv333_forward_keep_rows(v, x, w, ld, "bf16")
    tree = C.conv333_forward_keep_tree(v, x, w, ld, "fp32")[1].bfloat16()
    want = C.conv333_forward_pretree(v, x.double(), tree.double(), w.double(), ld, "fp32")[0]
    assert C.tc_error_flag() == 0
    assert float((got - want).norm() / want.norm()) <= 27 * ((cin + 15) // 16) * 2.0 ** -23
    bias = torch.randn(cout, device="cuda")
    assert torch.equal(C.conv333_forward_keep_rows(v, x, w, ld, "bf16", bias)[0], got + bias.view(1, -1, 1))
