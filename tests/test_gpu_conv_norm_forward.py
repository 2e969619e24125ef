"""`conv_norm` over two tensors and without gradients, against the concatenation and the two functions: the same kernels over the same values, so the forward pass
and, where a backward pass follows, the gradients are equal bit for bit."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


def _setup(names, dl, pad):
    import pyapr
    arrays = [H.blob_arrays((64, 64, 128), 40, 5) if name == "volume" else H.arrays(name) for name in names]
    aprs = [pyapr.apr_from_arrays(a) for a in arrays]
    for a in aprs:
        a.init_cuda()
    n = max(int(pyapr.aprnet.utils.number_particles(a, dl)) for a in aprs) + pad
    return aprs, n, torch.full((len(aprs),), dl, dtype=torch.int32)


def _modules(cin, cout, groups, precision, affine=True):
    from pyapr.aprnet import cuda as ops
    conv = ops.APRConv(cin, cout, nstencils=2, bias=False, precision=precision).cuda()
    norm = ops.GroupNormReLU(groups, cout, affine=affine).cuda()
    if affine:
        with torch.no_grad():
            norm.weight.uniform_(0.5, 1.5); norm.bias.uniform_(-0.5, 0.5)
    return conv, norm


# channels in front: a tile of the packing and less, none of a multiple of four (written out then); items of one size, of two, entries behind all of them; more
# entries behind an item than a tile of the normalisation has
@pytest.mark.parametrize("front,behind,cout,groups", [(32, 32, 32, 32), (4, 1, 8, 2), (36, 29, 17, 1), (64, 64, 64, 16), (33, 31, 40, 40), (0, 6, 32, 32), (0, 2, 16, 16)])
@pytest.mark.parametrize("names,dl,pad", [(["odd"], 0, 0), (["odd", "ref_shape"], 0, 0), (["volume", "odd", "cube32"], 1, 5), (["cube16"], 1, 3000)])
@pytest.mark.parametrize("precision", ["bf16", "fp32"])
def test_forward_without_gradients(front, behind, cout, groups, names, dl, pad, precision):
    from pyapr.aprnet import cuda as ops
    aprs, n, ld = _setup(names, dl, pad)
    torch.manual_seed(front + behind)
    conv, norm = _modules(front + behind, cout, groups, precision, affine=groups > 1)
    x = torch.randn(len(aprs), behind, n, device="cuda")
    skip = torch.randn(len(aprs), front, n, device="cuda") if front else None
    with torch.no_grad():
        want = norm(conv(x if skip is None else torch.cat([skip, x], 1), aprs, ld))
        # memory that was in use: nothing may come from entries that are not written
        junk = torch.full((4 * want.numel(),), float("nan"), device="cuda"); del junk
        got = ops.conv_norm(conv, norm, x, aprs, ld, skip)
    assert torch.equal(got, want)


@pytest.mark.parametrize("front,behind,cout", [(32, 32, 32), (4, 13, 40), (64, 64, 64), (6, 10, 16)])
@pytest.mark.parametrize("first,second", [(True, True), (True, False), (False, True)])
def test_gradients_of_two_inputs(front, behind, cout, first, second):
    from pyapr.aprnet import cuda as ops
    from _pyaprwrapper.aprnet import cuda as C
    aprs, n, ld = _setup(["volume"], 0, 0)
    torch.manual_seed(cout)
    conv, norm = _modules(front + behind, cout, cout, "bf16")
    x0, x1, g = torch.randn(1, behind, n, device="cuda"), torch.randn(1, front, n, device="cuda"), torch.randn(1, cout, n, device="cuda")
    res = []
    for pair in (False, True):
        conv.zero_grad(set_to_none=True); norm.zero_grad(set_to_none=True)
        x, skip = x0.clone().requires_grad_(second), x1.clone().requires_grad_(first)
        y = ops.conv_norm(conv, norm, x, aprs, ld, skip) if pair else ops.conv_norm(conv, norm, torch.cat([skip, x], 1), aprs, ld)
        y.backward(g)
        res.append([y.detach(), x.grad, skip.grad, conv.weight.grad, norm.weight.grad, norm.bias.grad])
    assert C.tc_error_flag() == 0
    for u, v in zip(*res):
        assert (u is None and v is None) or torch.equal(u, v)


@pytest.mark.parametrize("wanted", [False, True])
def test_pooling_without_indices(wanted):
    from pyapr.aprnet import cuda as ops
    aprs, n, ld = _setup(["odd", "ref_shape"], 0, 0)
    x = torch.randn(2, 5, n, device="cuda")
    want = ops.MaxPool()(x.clone().requires_grad_(True), aprs, ld.clone()).detach()
    got = ops.MaxPool()(x.requires_grad_(wanted), aprs, ld.clone())
    assert torch.equal(got.detach(), want) and got.requires_grad == wanted


@pytest.mark.parametrize("front,behind", [(33, 31), (6, 10), (1, 32), (32, 32), (0, 20)])
def test_training_is_one_function_at_any_split(front, behind):
    """A number of channels in front that the packing of two tensors does not take costs the concatenation, not the joint backward pass: the same bits as one tensor."""
    from pyapr.aprnet import cuda as ops
    aprs, n, ld = _setup(["volume"], 0, 0)
    torch.manual_seed(front)
    conv, norm = _modules(front + behind, 16, 4, "bf16")
    whole, g = torch.randn(1, front + behind, n, device="cuda"), torch.randn(1, 16, n, device="cuda")
    res = []
    for split in (False, True):
        conv.zero_grad(); norm.zero_grad()
        x = whole.clone().requires_grad_(True)
        y = ops.conv_norm(conv, norm, x[:, front:], aprs, ld, x[:, :front]) if split and front else ops.conv_norm(conv, norm, x, aprs, ld)
        assert "ConvGroupNormReLUFunction" in y.grad_fn.name()
        y.backward(g)
        res.append([y.detach(), x.grad] + [p.grad.clone() for m in (conv, norm) for p in m.parameters()])
    assert all(torch.equal(a, b) for a, b in zip(*res))


def test_no_channels_behind():
    """The tensor in front may be all of the input."""
    from pyapr.aprnet import cuda as ops
    aprs, n, ld = _setup(["odd"], 0, 0)
    conv, norm = _modules(8, 8, 2, "bf16")
    x = torch.randn(1, 8, n, device="cuda")
    with torch.no_grad():
        assert torch.equal(ops.conv_norm(conv, norm, x[:, 8:], aprs, ld, x), ops.conv_norm(conv, norm, x, aprs, ld))
