"""The fp32 row kernels against the fp64 oracle at the widths where their tiles change: output tiles of 8, 16, 32 and 64
channels, input blocks of 8, 16 and 32, remainders of each, a bias, and a batch padded beyond the valid entries.
Tolerance: fp32 sums over 27 * C products of unit scale, relative error <= 1e-5 (as in the other parity tests)."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(5, 8), (8, 9), (17, 16), (16, 31), (33, 32), (24, 65), (64, 48), (40, 64), (70, 5)])
def test_row_kernels_match_oracle(cin, cout, oracle):
    import pyapr
    from pyapr.aprnet import cuda as ops
    a = H.blob_arrays()
    b = H.arrays("odd")
    aprs, orcs = [], []
    for s in (a, b):
        apr = pyapr.apr_from_arrays(s)
        apr.init_cuda()
        aprs.append(apr)
        orcs.append(oracle.OracleAPR(s))
    dls = [1, 0]
    n = [o.number_parts(d) for o, d in zip(orcs, dls)]
    pad = max(n) + 7
    torch.manual_seed(3)
    conv = ops.APRConv(cin, cout, nstencils=2, precision="fp32").cuda()
    x = torch.randn(2, cin, pad, device="cuda", requires_grad=True)
    g = torch.randn(2, cout, pad, device="cuda")
    ld = torch.tensor(dls, dtype=torch.int32)
    out = conv(x, aprs, ld)
    out.backward(g)
    levels = max(s.level_max - s.level_min + 1 for s in (a, b))
    w = oracle.restrict333_forward(conv.weight.detach().cpu().double().numpy(), levels)
    bias = conv.bias.detach().cpu().double().numpy()[:, None]
    gw = 0.0
    for i, (o, d) in enumerate(zip(orcs, dls)):
        xi = x[i, :, :n[i]].detach().cpu().double().numpy()
        gi = g[i, :, :n[i]].cpu().double().numpy()
        assert H.rel_err(H.t2n(out[i, :, :n[i]]), o.conv333_forward(xi, w, d) + bias) <= 1e-5
        assert torch.equal(out[i, :, n[i]:], conv.bias.detach()[:, None].expand(-1, pad - n[i]))      # zero padding plus bias
        gi_ref, gw_ref = o.conv333_backward(xi, w, gi, d)
        assert H.rel_err(H.t2n(x.grad[i, :, :n[i]]), gi_ref) <= 1e-5
        assert not x.grad[i, :, n[i]:].any()
        gw = gw + gw_ref
    assert H.rel_err(H.t2n(conv.weight.grad), oracle.restrict333_backward(gw, 2)) <= 1e-5
    assert H.rel_err(H.t2n(conv.bias.grad), g.cpu().double().sum(dim=(0, 2)).numpy()) <= 1e-5
