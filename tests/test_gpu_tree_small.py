"""Tree fill of one tensor and of two that stand for their concatenation, where all levels are in the launch of the coarse ones (small structures) and where they are not."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["odd", "cube32", "ref_shape", "volume"])
@pytest.mark.parametrize("front,behind", [(4, 4), (8, 3), (4, 13), (32, 32)])
def test_two_tensors_as_their_concatenation(name, front, behind):
    """The means reach the packed rows behind the particles: the same bits from two tensors as from one."""
    import pyapr
    from pyapr.aprnet import cuda as ops
    apr = pyapr.apr_from_arrays(H.blob_arrays((64, 128, 128), 40, 11) if name == "volume" else H.arrays(name))
    apr.init_cuda()
    n, ld = int(pyapr.aprnet.utils.number_particles(apr, 0)), torch.zeros(1, dtype=torch.int32)
    torch.manual_seed(front + behind)
    x = torch.randn(1, front + behind, n, device="cuda")
    for precision in ("fp32", "bf16"):
        conv, norm = ops.APRConv(front + behind, 8, bias=False, precision=precision).cuda(), ops.GroupNormReLU(2, 8).cuda()
        with torch.no_grad():
            whole = ops.conv_norm(conv, norm, x, [apr], ld)
            assert torch.equal(ops.conv_norm(conv, norm, x[:, front:].contiguous(), [apr], ld, x[:, :front].contiguous()), whole)


@pytest.mark.parametrize("dtype,eps", [(torch.float32, 2.0 ** -24), (torch.float64, 2.0 ** -53)])
@pytest.mark.parametrize("channels", [1, 2, 5])
@pytest.mark.parametrize("name", ["cube16", "odd", "cube32", "ref_shape"])
def test_means_and_maxima_of_small_structures(name, channels, dtype, eps, oracle):
    """Against the oracle: maxima are copies; a mean takes eight additions and a product per level, each rounding at most `eps` of the largest value."""
    import pyapr
    a = H.arrays(name)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(channels)
    parts = torch.rand(channels, a.n_particles, device="cuda", dtype=dtype)
    host, o = H.t2n(parts).astype("float64"), oracle.OracleAPR(a)
    mean, best = H.t2n(pyapr.tree.fill_tree_mean(apr, parts)), H.t2n(pyapr.tree.fill_tree_max(apr, parts))
    want = o.fill_tree_mean(host, 0)
    assert abs(mean - want).max() <= 9 * a.level_max * eps
    for c in range(channels):
        assert (best[c] == o.fill_tree_max(host[c])).all()
