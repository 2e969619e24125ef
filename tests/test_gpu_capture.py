"""C ABI: after aprnet_plan_build and aprnet_edge_plan_build the convolutions of a new handle can be captured in a CUDA graph (nothing
synchronises or allocates outside the stream's order any more), and a replay gives what an ordinary call gives, bit for bit."""
import ctypes as C

import pytest
import torch

import helpers as H
from test_zz_no_alloc import _create, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["bf16", "fp32"])
@pytest.mark.parametrize("dl", [0, 1])
def test_convolution_in_a_graph(precision, dl):
    lib = _lib()
    for f in ("aprnet_tree_size", "aprnet_conv333_tc_workspace_bytes", "aprnet_conv333_tc_forward_workspace_bytes",
              "aprnet_conv333_tc_dw_partial_elems", "aprnet_conv333_partial_elems"):
        getattr(lib, f).restype = C.c_int64
    cin, cout, slots = 32, 40, 2
    a = H.blob_arrays()
    dev = torch.device("cuda:0")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    i64 = C.c_int64

    def buffers(h):
        n, t = int(lib.aprnet_number_parts(h, dl)), int(lib.aprnet_tree_size(h, dl))
        torch.manual_seed(7)
        b = dict(n=n, t=max(t, 1), x=torch.randn(cin, n, device=dev), g=torch.randn(cout, n, device=dev), w=torch.randn(slots, cout, cin, 27, device=dev) / 30,
                 out=torch.zeros(cout, n, device=dev), gin=torch.zeros(cin, n, device=dev), gw=torch.zeros(slots, cout, cin, 27, device=dev),
                 tree=torch.zeros(cin, max(t, 1), device=dev), gtree=torch.zeros(cin, max(t, 1), device=dev))
        ws = max(lib.aprnet_conv333_tc_workspace_bytes(h, dl, cin, cout, slots), lib.aprnet_conv333_tc_forward_workspace_bytes(h, dl, cin, cout, slots))
        b["ws"] = torch.zeros(ws, dtype=torch.uint8, device=dev)
        b["partial"] = torch.zeros(max(lib.aprnet_conv333_tc_dw_partial_elems(cin, cout), lib.aprnet_conv333_partial_elems(cin, cout)), device=dev)
        return b

    def launch(h, b):
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        n, t = i64(b["n"]), i64(b["t"])
        b["gw"].zero_()
        if precision == "bf16":
            rcs = [lib.aprnet_conv333_forward_tc(h, dl, cin, cout, slots, ptr(b["x"]), n, ptr(b["w"]), ptr(b["out"]), n, ptr(b["tree"]), t, ptr(b["ws"]), st),
                   lib.aprnet_conv333_backward_tc_rows(h, dl, cin, cout, slots, ptr(b["ws"]), ptr(b["g"]), n, ptr(b["w"]), ptr(b["gin"]), n, ptr(b["gw"]),
                                                       ptr(b["gtree"]), t, ptr(b["partial"]), ptr(b["ws"]), st)]
        else:
            rcs = [lib.aprnet_conv333_forward(h, dl, 0, cin, cout, slots, ptr(b["x"]), n, ptr(b["w"]), ptr(b["out"]), n, ptr(b["tree"]), t, st),
                   lib.aprnet_conv333_backward_weights(h, dl, 0, cin, cout, slots, ptr(b["x"]), n, ptr(b["tree"]), t, ptr(b["g"]), n, ptr(b["gw"]), ptr(b["partial"]), st),
                   lib.aprnet_conv333_backward_input(h, dl, 0, cin, cout, slots, ptr(b["g"]), n, ptr(b["w"]), ptr(b["gin"]), n, ptr(b["gtree"]), t, st)]
        assert rcs == [0] * len(rcs), lib.aprnet_last_error()

    first, h = _create(lib, a), _create(lib, a)
    try:
        launch(first, buffers(first))                       # the library is loaded, its error flag exists
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.aprnet_plan_build(h, dl, st) == 0 and lib.aprnet_edge_plan_build(h, dl, st) == 0
        b = buffers(h)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            launch(h, b)
        for k in ("out", "gin", "gw"):
            b[k].fill_(float("nan"))
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        got = {k: b[k].clone() for k in ("out", "gin", "gw")}
        launch(h, b)
        torch.cuda.synchronize()
        for k in got:
            assert torch.isfinite(got[k]).all() and torch.equal(got[k], b[k]), k
        del graph
    finally:
        torch.cuda.synchronize()
        lib.aprnet_apr_destroy(first)
        lib.aprnet_apr_destroy(h)
