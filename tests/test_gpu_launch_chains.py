"""Tree levels whose launches overlap: a level's kernel starts while the finer (adjoint: coarser) one still runs and waits only for what that one writes.
Calls that are queued one behind the other, on memory that the allocator hands round, give the bits of calls with the GPU idle in between, and so does a captured
sequence; values against the oracle (fp32 sums of at most eight children or one parent per level: relative 1e-6)."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 9])
@pytest.mark.parametrize("dl", [0, 1])
def test_levels_launched_behind_each_other(dl, channels, oracle):
    import pyapr
    from pyapr import synthetic
    from _pyaprwrapper.aprnet import cuda as C
    level_map = torch.full((64, 64, 64), 6, dtype=torch.int32)          # 32768 tree nodes at level 5: launches of their own around it
    level_map[8:40, 8:40, 8:40] = 7                                     # and as many at level 6
    a = synthetic.apr_from_level_map(level_map, (128, 128, 128))
    o = oracle.OracleAPR(a)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(1)
    n = o.number_parts(dl)
    xs = [torch.randn(channels, n, device="cuda") for _ in range(12)]
    gts = [torch.randn_like(C.fill_tree_mean(apr, xs[0], dl)) for _ in xs]

    def step(x, gt):
        return C.fill_tree_mean(apr, x, dl), C.fill_tree_mean_backward(apr, x, gt, dl)

    alone = []
    for x, gt in zip(xs, gts):
        torch.cuda.synchronize()
        alone.append(step(x, gt))
    torch.cuda.synchronize()
    assert H.rel_err(H.t2n(alone[0][0]), o.fill_tree_mean(H.t2n(xs[0]).astype(np.float64), dl)) <= 1e-6
    want = o.fill_tree_mean_backward(H.t2n(xs[0]).astype(np.float64), H.t2n(gts[0]).astype(np.float64), dl)
    assert H.rel_err(H.t2n(alone[0][1]), want) <= 1e-6
    for _ in range(3):
        queued = [step(x * 1, gt * 1) for x, gt in zip(xs, gts)]        # inputs that a kernel directly before has written, freed after the call
        for got, ref in zip(queued, alone):
            assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    x, gt = xs[0].clone(), gts[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step(x, gt)
    for i in (3, 7):
        x.copy_(xs[i])
        gt.copy_(gts[i])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured[0], alone[i][0]) and torch.equal(captured[1], alone[i][1])
