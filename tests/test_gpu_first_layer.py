"""First layers (at most four input channels) at the sizes where the forward kernel changes its shape, against the fp64 kernels: a warp yields
30 slots of the run plan and takes the y neighbours from the lanes beside, a block's tile is 120 slots, and a block takes several tiles where
there are many.  At most 4 x 27 products and a
bias are added in fp32, and restricting a stencil keeps the sum of its magnitudes at most that of the original: the result is within
110 x 2^-24 of 108 max|x| max|w| + max|b|; the roundings of the restricted stencils and the tree means themselves (at most 27 + 8
terms per level, fewer than eight levels) make it four times that."""
import math

import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


def _check(a, cin, cout):
    import pyapr
    from pyapr.aprnet import cuda as ops
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    n = int(pyapr.aprnet.utils.number_particles(apr, 0))
    torch.manual_seed(cin)
    conv = ops.APRConv(cin, cout, nstencils=1, precision="fp32").cuda()
    x, ld = torch.randn(1, cin, n, device="cuda"), torch.zeros(1, dtype=torch.int32)
    with torch.no_grad():
        out = conv(x, [apr], ld).double()
        bound = 108 * x.abs().max() * conv.weight.abs().max() + (conv.bias.abs().max() if conv.bias is not None else 0)
        want = conv.double()(x.double(), [apr], ld)
    assert float((out - want).abs().max()) <= float(bound) * 4 * 110 * 2.0 ** -24


@pytest.mark.parametrize("shape,blobs", [((17, 33, 41), 3), ((64, 128, 128), 40), ((128, 256, 256), 300)])
@pytest.mark.parametrize("cin,cout", [(1, 32), (2, 40), (3, 7), (4, 64)])
def test_first_layer_forward(shape, blobs, cin, cout):
    _check(H.blob_arrays(shape, blobs, 5), cin, cout)


# one row of cells of the finest level, which is as many slots and two more: the ends of a warp's 30 and of a block's 120 slots
@pytest.mark.parametrize("cells", [26, 27, 28, 29, 57, 58, 59, 117, 118, 119, 237, 238, 239])
@pytest.mark.parametrize("cin,cout", [(1, 32), (2, 40), (3, 7), (4, 64)])
def test_ends_of_a_run(cells, cin, cout):
    from pyapr import synthetic
    top = math.ceil(math.log2(cells))
    a = synthetic.apr_from_level_map(torch.full((1, 1, (cells + 1) // 2), top, dtype=torch.int32), (1, 1, cells))
    assert a.n_particles == cells
    _check(a, cin, cout)
