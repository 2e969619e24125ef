"""The split form of the fp32 backward pass (z-slabs) on a structure beyond the 32-bit edge ids of the edge plan (more than 79.5 M
locations): the cross-level part is scattered, the tree gradient stays unfolded.  Against the float64 kernels, relative 1e-5 (fp32 sums)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_split_backward_beyond_the_edge_plan():
    import pyapr
    from pyapr import synthetic
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    edge = 440
    level_map = torch.full((edge // 2,) * 3, 9, dtype=torch.int32, device="cuda")
    level_map[:40, :40, :40] = 7                    # a coarser corner: edges between levels
    a = synthetic.apr_from_level_map(level_map, (edge,) * 3)
    n = a.n_particles
    assert 27 * n + 1 >= 2 ** 31
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    v, ld, L = APRPtrVector([apr]), torch.zeros(1, dtype=torch.int32), a.level_max - a.level_min + 1
    torch.manual_seed(4)
    x = torch.randn(1, 1, n, device="cuda")
    g = torch.randn(1, 1, n, device="cuda")
    w = torch.randn(L, 1, 1, 3, 3, 3, device="cuda")
    tree = C.conv333_forward_keep_tree(v, x, w, ld, "fp32")[1]
    none = torch.empty(0, dtype=torch.uint8, device="cuda")
    got = C.conv333_backward_pretree(v, x, tree, none, w, g, ld, True)
    want = C.conv333_backward_pretree(v, x.double(), tree.double(), none, w.double(), g.double(), ld, True)
    for a_, b_ in zip(got, want):
        assert b_.norm() > 0 and float((a_.double() - b_).norm() / b_.norm()) <= 1e-5


def test_split_backward_without_input_gradient_returns_zeros():
    """fp32: an input gradient that is not wanted comes back as zeros, like the tree gradient."""
    import helpers as H
    import pyapr
    from _pyaprwrapper.aprnet import cuda as C
    from _pyaprwrapper.data_containers import APRPtrVector
    a = H.blob_arrays()
    apr = pyapr.apr_from_arrays(a)
    apr.init_cuda()
    v, ld, n = APRPtrVector([apr]), torch.zeros(1, dtype=torch.int32), a.n_particles
    x, g = torch.randn(1, 6, n, device="cuda"), torch.randn(1, 5, n, device="cuda")
    w = torch.randn(a.level_max - a.level_min + 1, 5, 6, 3, 3, 3, device="cuda")
    tree = C.conv333_forward_keep_tree(v, x, w, ld, "fp32")[1]
    gi, gt, _ = C.conv333_backward_pretree(v, x, tree, torch.empty(0, dtype=torch.uint8, device="cuda"), w, g, ld, False)
    assert gi.shape == x.shape and not gi.any() and gt.shape == tree.shape and not gt.any()
