"""`conv_norm` (convolution, GroupNorm and ReLU as one function, the gradient between them only as packed rows) against the two functions."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


# channels: multiples of the 32 and 8 of a tile and none; groups of one and of several channels; few and many partial sums of a group;
# particles behind the structure's own; fully or not at all affine
@pytest.mark.parametrize("cin,cout,groups,pad,affine", [(32, 32, 32, 0, True), (8, 40, 5, 3, True), (33, 17, 1, 131, False), (64, 72, 36, 1, True), (5, 128, 128, 0, True)])
@pytest.mark.parametrize("name", ["odd", "ref_shape", "volume"])
def test_conv_norm_equals_the_two_functions(name, cin, cout, groups, pad, affine):
    import pyapr
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    a = H.blob_arrays((64, 64, 128), 40, 5) if name == "volume" else H.arrays(name)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    for dl in sorted({0, min(1, H.max_dl(a))}):
        n = int(pyapr.aprnet.utils.number_particles(apr, dl))
        torch.manual_seed(3)
        conv = ops.APRConv(cin, cout, nstencils=2, bias=False, precision="bf16").cuda()
        norm = ops.GroupNormReLU(groups, cout, affine=affine).cuda()
        if affine:
            with torch.no_grad():
                norm.weight.uniform_(0.5, 1.5); norm.bias.uniform_(-0.5, 0.5)
        x = torch.randn(1, cin, n + pad, device="cuda")
        g = torch.randn(1, cout, n + pad, device="cuda")
        ld = torch.full((1,), dl, dtype=torch.int32)
        res = []
        for joint in (False, True):
            conv.zero_grad(set_to_none=True); norm.zero_grad(set_to_none=True)
            xi = x.clone().requires_grad_(True)
            y = ops.conv_norm(conv, norm, xi, [apr], ld) if joint else norm(conv(xi, [apr], ld))
            assert (type(y.grad_fn).__name__ == "ConvGroupNormReLUFunctionBackward") == joint
            y.backward(g)
            res.append([y.detach(), xi.grad, conv.weight.grad] + [p.grad for p in norm.parameters()])
        assert C.tc_error_flag() == 0
        assert torch.equal(res[0][0], res[1][0])
        # the gradient between the two is the same expression in both kernels; where the compilers' contractions differ in its last bit (2^-24), a
        # rounding to bf16 (2^-9) may differ for one value in 2^15
        for u, v in zip(res[0][1:], res[1][1:]):
            assert float((u - v).norm()) <= 1e-4 * float(u.norm())


def test_conv_norm_calls_modules_that_are_observed():
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.arrays("odd")
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    conv, norm = ops.APRConv(8, 8, bias=False, precision="bf16").cuda(), ops.GroupNormReLU(8, 8).cuda()
    x, ld = torch.randn(1, 8, a.n_particles, device="cuda", requires_grad=True), torch.zeros(1, dtype=torch.int32)
    seen = []
    handle = conv.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    ops.conv_norm(conv, norm, x, [apr], ld)
    handle.remove()
    assert len(seen) == 1
    for p, other in (("fp32", norm), ("bf16", torch.nn.GroupNorm(8, 8).cuda())):
        conv.precision = p
        assert type(ops.conv_norm(conv, other, x, [apr], ld).grad_fn).__name__ != "ConvGroupNormReLUFunctionBackward"


@pytest.mark.parametrize("affine", [True, False])
def test_a_convolution_that_is_not_trained_keeps_nothing(affine):
    """Input and weights without a gradient: the two functions, whose convolution has no backward pass and keeps no rows for one."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays((64, 64, 128), 40, 5)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    conv, norm = ops.APRConv(32, 32, bias=False, precision="bf16").cuda(), ops.GroupNormReLU(32, 32, affine=affine).cuda()
    conv.requires_grad_(False)
    x, ld = torch.randn(1, 32, a.n_particles, device="cuda"), torch.zeros(1, dtype=torch.int32)
    g = torch.randn(1, 32, a.n_particles, device="cuda")
    res = []
    for call in (lambda: norm(conv(x, [apr], ld)), lambda: ops.conv_norm(conv, norm, x, [apr], ld)):
        norm.zero_grad(set_to_none=True)
        y = call()
        del y
        before = torch.cuda.memory_allocated()
        y = call()
        held = torch.cuda.memory_allocated() - before
        assert y.requires_grad == affine
        if affine:
            assert type(y.grad_fn).__name__ == "GroupNormReLUFunctionBackward"
            y.backward(g)
        res.append((held, [y.detach()] + [p.grad for p in norm.parameters()]))
    assert res[1][0] <= res[0][0]
    assert all(torch.equal(u, v) for u, v in zip(res[0][1], res[1][1]))
