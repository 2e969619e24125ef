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
