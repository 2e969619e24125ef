"""A bias that the kernels do not take as it lies (strided, of another type, one value for all channels) behaves like a torch addition:
same result type, values and padding; the gradient is the sum of grad_output over batch and locations."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [(3, 3, 3), (1, 1, 1)])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("kind", ["strided", "float64", "bfloat16", "one value", "expanded"])
def test_unusual_bias(kernel, precision, kind):
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays()
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(5)
    cin, cout, n = 9, 12, a.n_particles + 3                # padded beyond the valid entries
    conv = ops.APRConv(cin, cout, kernel_size=kernel, precision=precision).cuda()
    bare = ops.APRConv(cin, cout, kernel_size=kernel, precision=precision, bias=False).cuda()
    bare.weight.data.copy_(conv.weight.data)
    b = {"strided": torch.randn(2 * cout, device="cuda")[::2], "float64": torch.randn(cout, device="cuda", dtype=torch.float64),
         "bfloat16": torch.randn(cout, device="cuda").bfloat16(), "one value": torch.randn(1, device="cuda"),
         "expanded": torch.randn(1, device="cuda").expand(cout)}[kind]
    conv.bias = torch.nn.Parameter(b, requires_grad=kind != "one value")
    x = torch.randn(1, cin, n, device="cuda")
    ld = torch.zeros(1, dtype=torch.int32)
    got, want = conv(x, [apr], ld), bare(x, [apr], ld) + b.view(1, -1, 1)
    assert got.dtype == want.dtype and torch.equal(got, want)
    if conv.bias.requires_grad and kind != "float64":        # (the kernels take no float64 gradient of float32 features)
        g = torch.randn_like(got)
        got.backward(g)
        want = g.double().sum(dim=(0, 2))
        # fp32 sums of some 10^4 terms of unit scale; a bfloat16 gradient is rounded once more (2^-9 of it)
        assert bool(((conv.bias.grad.double() - want).abs() <= 1e-2 + (2.0 ** -8 if kind == "bfloat16" else 0) * want.abs()).all())


@pytest.mark.parametrize("name", ["odd", "plane", "volume"])
@pytest.mark.parametrize("cin,cout", [(8, 8), (5, 33), (33, 64), (16, 200)])
@pytest.mark.parametrize("frozen_input", [False, True])
def test_bias_gradient_is_taken_along(name, cin, cout, frozen_input):
    """3x3x3, bf16: the sums of the gradient that is packed.  Four fp32 values are added in two roundings, all else in double precision, one more rounding at the
    end: |error| <= 3 * 2^-24 of the sum of magnitudes.  A padded item and a batch are summed by torch, also behind the particles: 2^-16."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays((64, 128, 128), 40, 11) if name == "volume" else H.arrays(name)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(cout)
    conv = ops.APRConv(cin, cout, nstencils=2, precision="bf16").cuda()
    bare = ops.APRConv(cin, cout, nstencils=2, precision="bf16", bias=False).cuda()
    bare.weight.data.copy_(conv.weight.data)
    for batch, pad in ((1, 0), (1, 3), (2, 0)):
        n = a.n_particles + pad
        x, g, ld = torch.randn(batch, cin, n, device="cuda"), torch.randn(batch, cout, n, device="cuda"), torch.zeros(batch, dtype=torch.int32)
        grads = []
        for m in (conv, bare):
            m.zero_grad(set_to_none=True)
            xi = x.clone().requires_grad_(not frozen_input)
            m(xi, [apr] * batch, ld).backward(g)
            grads.append([m.weight.grad, xi.grad])
        want, size = g.double().sum(dim=(0, 2)), g.double().abs().sum(dim=(0, 2))
        assert bool(((conv.bias.grad.double() - want).abs() <= size * (3 * 2.0 ** -24 if (batch, pad) == (1, 0) else 2.0 ** -16)).all())
        assert torch.equal(grads[0][0], grads[1][0]) and (frozen_input or torch.equal(grads[0][1], grads[1][1]))
