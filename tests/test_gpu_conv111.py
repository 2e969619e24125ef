"""1x1x1 layers on the tensor cores at the edges of their tiles (pairs of 128 locations, pieces of 16 channels, 128-byte lines): with
one stencil the layer is one matrix product over all locations.  Operands are exact in bf16 and at most 256 products are added in
fp32, each rounding at most 2^-24 of the sum of magnitudes so far: |error| <= 2^-16 of that sum for the forward pass and the input
gradient.  The weight gradient adds over all locations, in blocks: 2-norm error at most 1e-5, the rounding errors of random sign."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu

WIDTHS = [(8, 8), (16, 17), (24, 16), (33, 40), (64, 128), (130, 72), (256, 128), (128, 250)]


@pytest.mark.parametrize("name", ["blob", "odd", "many"])
@pytest.mark.parametrize("cin,cout", WIDTHS)
def test_conv111_edges(name, cin, cout):
    import pyapr
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    a = H.blob_arrays((64, 128, 128), 40, 11) if name == "many" else (H.arrays(name) if name in H.APR_CASES else H.blob_arrays())
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(cin * 300 + cout)
    exact = lambda *s: torch.randn(*s, device="cuda").bfloat16().float()
    for dl in range(0, min(H.max_dl(a), 2) + 1):
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        conv = ops.APRConv(cin, cout, nstencils=1, kernel_size=(1, 1, 1), precision="bf16").cuda()
        with torch.no_grad():
            conv.weight.copy_(exact(*conv.weight.shape))
        x, g = exact(1, cin, n).requires_grad_(True), exact(1, cout, n)
        out = conv(x, [apr], torch.full((1,), dl, dtype=torch.int32))
        out.backward(g)
        assert C.tc_error_flag() == 0
        w, xd, gd = conv.weight.detach().double().reshape(cout, cin), x.detach()[0].double(), g[0].double()
        want, size = w @ xd, w.abs() @ xd.abs()
        if conv.bias is not None:
            b = conv.bias.detach().double().reshape(-1, 1)
            want, size = want + b, size + b.abs()
        assert bool(((out.detach()[0].double() - want).abs() <= size * 2.0 ** -16).all()), dl
        want, size = w.t() @ gd, w.t().abs() @ gd.abs()
        assert bool(((x.grad[0].double() - want).abs() <= size * 2.0 ** -16).all()), dl
        want = gd @ xd.t()
        assert float((conv.weight.grad.double().reshape(cout, cin) - want).norm() / want.norm()) <= 1e-5, dl


@pytest.mark.parametrize("cin,cout", [(8, 8), (17, 16), (16, 33), (64, 24), (100, 128), (24, 200), (128, 31), (64, 256)])
def test_conv111_joint_gradients(cin, cout):
    """All gradients of a layer with a stencil per level and a bias, one item and a padded batch.  A bias gradient adds the fp32 values of at most 14 k locations
    in chains of at most 64 after 7 halvings, the blocks' sums in chains of at most 20: |error| <= (64 + 7 + 20 + 8) 2^-24 < 2^-17 of the sum of magnitudes."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    arrays = [H.blob_arrays((64, 128, 128), 40, 11), H.arrays("odd")]
    aprs = [pyapr.apr_from_arrays(a) for a in arrays]
    for a in aprs:
        a.init_cuda()
    torch.manual_seed(cin + 1000 * cout)
    exact = lambda *s: torch.randn(*s, device="cuda").bfloat16().float()
    counts = [int(pyapr.aprnet.utils.number_particles(a, 0)) for a in aprs]
    for items in ([0], [1], [0, 1]):
        n = max(counts[k] for k in items)
        conv = ops.APRConv(cin, cout, nstencils=3, kernel_size=(1, 1, 1), precision="bf16").cuda()
        with torch.no_grad():
            conv.weight.copy_(exact(*conv.weight.shape))
        x, g = exact(len(items), cin, n).requires_grad_(True), torch.randn(len(items), cout, n, device="cuda")
        gb = g.bfloat16().float()
        conv(x, [aprs[k] for k in items], torch.zeros(len(items), dtype=torch.int32)).backward(g)
        want_w = torch.zeros(3, cout, cin, device="cuda", dtype=torch.double)
        for b, k in enumerate(items):
            a, begin, row = arrays[k], 0, 0
            for level in range(a.level_min, a.level_max + 1):
                row += a.dims[level][0] * a.dims[level][1]
                end = int(a.row_ptr[row])
                slot = min(a.level_max - level, 2)
                gd, xd, w = gb[b, :, begin:end].double(), x.detach()[b, :, begin:end].double(), conv.weight.detach()[slot].double().reshape(cout, cin)
                size = w.t().abs() @ gd.abs()
                assert bool(((x.grad[b, :, begin:end].double() - w.t() @ gd).abs() <= size * 2.0 ** -16).all()), (items, level)
                want_w[slot] += gd @ xd.t()
                begin = end
            assert end == counts[k] and bool((x.grad[b, :, end:] == 0).all())
        assert float((conv.weight.grad.double().reshape(3, cout, cin) - want_w).norm() / want_w.norm()) <= 1e-5
        want = g.double().sum(dim=(0, 2))
        assert bool(((conv.bias.grad.double() - want).abs() <= g.double().abs().sum(dim=(0, 2)) * 2.0 ** -17).all())


def test_conv111_bias_sums_of_equal_values_are_exact():
    """2^21 locations, so that a block adds more than fifty tiles: 128 equal values of a tile add up exactly in fp32, the tiles exactly in double precision (24 + 21
    bits), and the result is a float times a power of two.  Chains in fp32 round it off (mantissas chosen so that each addition loses nearly half a bit)."""
    import pyapr
    from pyapr import synthetic
    from pyapr.aprnet import cuda as ops
    apr = pyapr.apr_from_arrays(synthetic.apr_from_level_map(torch.full((64, 64, 64), 7, dtype=torch.int16), (128, 128, 128)))
    apr.init_cuda()
    n = int(pyapr.aprnet.utils.number_particles(apr, 0))
    assert n == 2 ** 21
    conv = ops.APRConv(32, 8, nstencils=1, kernel_size=(1, 1, 1), precision="bf16").cuda()
    value = 1 + torch.tensor([912, 783, 752, 686352, 7748513, 31, 127, 8191], device="cuda").float() * 2.0 ** -23
    x, g = torch.zeros(1, 32, n, device="cuda"), value.view(1, -1, 1).repeat(1, 1, n)
    conv(x, [apr], torch.zeros(1, dtype=torch.int32)).backward(g)
    assert torch.equal(conv.bias.grad, value * 2.0 ** 21)
