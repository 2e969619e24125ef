"""Tree fill on structures whose finest level is rare: a coarser tree level then holds far more nodes than a finer one.  Only the
coarsest levels that are all small share a launch; values against the oracle (the mean: fp32 sums of at most eight children per level,
relative 1e-6; the maximum: exact)."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 5])
def test_rare_finest_level(channels, oracle):
    import pyapr
    from pyapr import synthetic
    from _pyaprwrapper.aprnet import cuda as C
    level_map = torch.full((64, 64, 64), 6, dtype=torch.int32)          # cells of level 6 everywhere: 32768 tree nodes at level 5,
    level_map[30:32, 30:32, 30:32] = 7                                  # and a spot of level 7: a handful at level 6
    a = synthetic.apr_from_level_map(level_map, (128, 128, 128))
    o = oracle.OracleAPR(a)
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    torch.manual_seed(1)
    x = torch.randn(channels, a.n_particles, device="cuda")
    for name, fill, ref in (("tree_mean_fwd", pyapr.tree.fill_tree_mean, lambda v: o.fill_tree_mean(v, 0)),
                            ("tree_max", pyapr.tree.fill_tree_max, lambda v: np.stack([o.fill_tree_max(c) for c in v]))):
        fill(apr, x)
        torch.cuda.synchronize()
        C.profile_read()
        C.profile_enable(True)
        got = fill(apr, x)
        torch.cuda.synchronize()
        C.profile_enable(False)
        # a launch for level 6 (few nodes), one for level 5 (32768), one for the levels 0 to 4 (at most 4096 each)
        assert C.profile_read()[name][0] == 3
        want = ref(x.cpu().double().numpy())
        assert H.rel_err(H.t2n(got), want) <= (1e-6 if name == "tree_mean_fwd" else 0)
