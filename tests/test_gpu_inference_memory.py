"""Without gradients a 3x3x3 layer holds the scratch of one batch item, not the packed rows of the batch."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("grad", ["no_grad", "nothing requires grad"])
def test_scratch_of_one_item(precision, grad):
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays((64, 128, 128), 40, 11)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(6)
    batch, c, n = 8, 32, a.n_particles
    conv = ops.APRConv(c, c, precision=precision).cuda()
    x = torch.randn(batch, c, n, device="cuda")
    ld = torch.zeros(batch, dtype=torch.int32)
    want = conv(x, [apr] * batch, ld).detach()
    if grad != "no_grad":
        conv.requires_grad_(False)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    with torch.set_grad_enabled(grad != "no_grad"):
        got = conv(x, [apr] * batch, ld)
    assert torch.equal(got, want) and not got.requires_grad
    item = 4 * c * (n + a.n_tree + 1)                     # packed rows of an item in fp32; tree means and packed weights are less
    assert torch.cuda.max_memory_allocated() - before <= got.numel() * 4 + 2 * item
