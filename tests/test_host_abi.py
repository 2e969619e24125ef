"""Host logic of the C ABI that needs no GPU, with handles and tables that are made up.

Device check: every convolution entry point checks that the current device is the handle's before it launches or copies anything.
Without a GPU the check is the one call that fails with "no current CUDA device"; an entry point that got past it would report its
first launch or copy instead.  (On a GPU the same calls would reach kernels with the made-up pointers.)

Cross-level input gradient: the sums per (target, tap) go through a bounded workspace in passes; no width may be refused.

Row numbers: the kernels hold them in 32 bits; structures beyond that are refused when a plan is built."""
import ctypes as C
import os
import re
import subprocess

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "apr-cnn_b200")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def helper(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    out = str(tmp_path_factory.mktemp("host") / "helper.so")
    subprocess.check_call([NVCC, "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                           os.path.join(ROOT, "tests", "host_helper.cu"), "-o", out])
    C.CDLL(os.path.join(PKG, "libaprnet_b200.so"), mode=C.RTLD_GLOBAL)
    helper = C.CDLL(out)
    helper.fake_handle.restype = C.c_void_p
    helper.vrow_worst_pass.restype = helper.vrow_chunk.restype = C.c_longlong
    return helper


@pytest.fixture(scope="module")
def lib(helper):
    lib = C.CDLL(os.path.join(PKG, "libaprnet_b200.so"), mode=C.RTLD_GLOBAL)
    lib.aprnet_last_error.restype = C.c_char_p
    lib.aprnet_edge_workspace_bytes.restype = lib.aprnet_conv333_rows_backward_workspace_bytes.restype = C.c_int64
    return lib, C.c_void_p(helper.fake_handle(3))


p, n = C.c_void_p(0x1000), C.c_int64(64)          # never dereferenced on the host
i = C.c_int
CALLS = {
    "aprnet_plan_build": (i(0), None),
    "aprnet_run_plan_build": (i(0), None),
    "aprnet_edge_plan_build": (i(0), None),
    "aprnet_conv333_forward": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, None),
    "aprnet_conv333_forward_pretree": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, None),
    "aprnet_conv333_backward_input": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, None),
    "aprnet_conv333_backward_input_pretree": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, None),
    "aprnet_conv333_backward_input_cross_level": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, None),
    "aprnet_conv333_backward_weights": (i(0), i(0), i(8), i(8), i(1), p, n, p, n, p, n, p, p, None),
    "aprnet_conv333_rows_forward": (i(0), i(0), i(8), i(8), i(1), p, n, p, None, p, n, p, n, i(1), p, None),
    "aprnet_conv333_rows_forward_pair": (i(0), i(1), i(8), i(8), i(1), p, n, i(4), p, n, p, None, p, n, p, n, p, None),
    "aprnet_conv333_rows_pack": (i(0), i(1), i(8), p, n, p, n, i(1), p, None),
    "aprnet_conv333_rows_backward": (i(0), i(1), i(8), i(8), i(1), p, p, n, p, p, n, p, i(0), p, n, i(1), p, p, None),
    "aprnet_conv333_rows_backward_bias": (i(0), i(8), i(8), i(1), p, p, n, p, p, n, p, p, n, p, p, p, None),
    "aprnet_conv333_forward_tc": (i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, p, None),
    "aprnet_conv333_forward_tc_pretree": (i(0), i(8), i(8), i(1), p, n, p, p, n, p, n, p, None),
    "aprnet_conv333_backward_tc": (i(0), i(8), i(8), i(1), p, n, p, n, p, p, p, p, i(1), p, n, p, p, None),
    "aprnet_conv333_backward_tc_rows": (i(0), i(8), i(8), i(1), p, p, n, p, p, n, p, p, n, p, p, None),
    "aprnet_conv333_backward_tc_rows_pretree": (i(0), i(8), i(8), i(1), p, p, n, p, p, n, p, p, n, p, p, None),
    "aprnet_conv333_backward_weights_tc": (i(0), i(8), i(8), i(1), p, i(16), p, i(16), p, p, None),
    "aprnet_conv333_backward_input_cross_level_tc": (i(0), i(8), i(8), i(1), p, i(16), p, p, n, p, n, p, p, n, None),
    "aprnet_conv111_forward": (i(0), i(0), i(8), i(8), i(1), p, n, p, p, n, None),
    "aprnet_conv111_forward_tc": (i(0), i(8), i(8), i(1), p, n, p, p, n, None),
    "aprnet_conv111_backward_tc": (i(0), i(8), i(8), i(1), p, n, p, n, p, p, n, p, p, p, C.c_int64(1 << 20), None),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_refused_before_anything_is_launched(lib, name):
    if torch.cuda.is_available():
        pytest.skip("with a GPU a missing check would launch kernels on made-up pointers")
    lib, handle = lib
    assert getattr(lib, name)(handle, *CALLS[name]) < 0
    assert lib.aprnet_last_error() == b"no current CUDA device"


@pytest.mark.parametrize("cout", [1, 64, 500, 512, 1024, 2048, 5000, 65536])
def test_cross_level_passes_fit_their_workspace(helper, lib, cout):
    lib, handle = lib
    for row in ((cout + 3) // 4 * 16, (cout + 15) // 16 * 32):                  # packed rows: fp32, bf16
        for n in (0, 1, 65535, 65536, 65537, 3 << 20, 4 << 20, (4 << 20) + 1, 40_000_000):
            assert helper.vrow_worst_pass(C.c_longlong(n), C.c_longlong(row)) <= 0, (row, n)
    helper.set_vrows(handle, C.c_longlong(40_000_000))
    # the workspaces that the library reports hold a chunk of the plan at any width
    assert lib.aprnet_edge_workspace_bytes(handle, 0, cout) >= helper.vrow_chunk() * ((cout + 15) // 16 * 32)
    assert lib.aprnet_conv333_rows_backward_workspace_bytes(handle, 0, 0, 8, cout, 1, 1) >= helper.vrow_chunk() * ((cout + 3) // 4 * 16)


@pytest.mark.parametrize("particles,nodes,over", [(16, 2, 0), (2 ** 31 - 1000, 998, 0), (2 ** 31 - 1000, 999, 1), (2 ** 31 - 3, 2 ** 31 - 3, 1)])
def test_row_numbers_fit_32_bits(helper, lib, particles, nodes, over):
    lib, handle = lib
    assert helper.rows_overflow(handle, C.c_longlong(particles), C.c_longlong(nodes)) == over
    if over:
        assert b"32-bit row numbers" in lib.aprnet_last_error()


@pytest.mark.parametrize("width,forward,per_sm", [(64, 1, 3), (64, 0, 2), (32, 1, 4), (32, 0, 3), (16, 1, 4), (16, 0, 3), (8, 1, 4), (8, 0, 3)])
def test_few_blocks_of_an_fp32_gather(helper, width, forward, per_sm):
    """One location per lane is the faster form as long as it puts at most `per_sm` of its blocks, four for one, on each of 148 SMs."""
    assert helper.f32_few_blocks(width, forward) * 4 == per_sm * 148


@pytest.mark.parametrize("nt,blocks", [(32, 4), (64, 2), (128, 2)])
def test_tallest_tile_over_runs(helper, nt, blocks):
    """Whatever a stage holds: with roles that branch per warp, taller tiles are slower for every number of source channels."""
    assert helper.run_max_height(nt) == blocks


def test_painting_needs_no_workspace(lib):
    """Cells to image: a null workspace is no bad argument (the device check comes after the arguments'); image to cells uses one."""
    if torch.cuda.is_available():
        pytest.skip("with a GPU the call would reach kernels with the made-up pointers")
    lib, handle = lib
    assert lib.aprnet_cells_to_image(handle, i(0), i(0), i(2), p, n, p, i(0), None, None) < 0
    assert lib.aprnet_last_error() == b"no current CUDA device"
    assert lib.aprnet_image_to_cells(handle, i(0), i(0), i(2), p, p, n, i(0), None, None) < 0
    assert b"workspace" in lib.aprnet_last_error()


def test_every_compiled_tile_over_runs_is_reached(helper):
    """The variants of the run kernel are those that the choice of a tile's height can ask for."""
    source = open(os.path.join(PKG, "csrc", "conv333_tc_runs.cu")).read()
    cases = [tuple(int(v) for v in c.split(",")) for c in re.findall(r"RUN_CASE\(((?:\d+, ){4}\d+)\)", source)]
    assert cases and {(nt, ks, order): max(h for a, b, c, h, _ in cases if (a, b, c) == (nt, ks, order)) for nt, ks, order, _, _ in cases} == {
        (nt, ks, order): helper.run_max_height(nt) for nt, ks, order, _, _ in cases}


@pytest.mark.parametrize("width,source,blocks,many", [(64, 8, 444, 0), (64, 8, 445, 1), (64, 128, 148, 0), (32, 16, 100000, 0), (32, 20, 444, 0), (32, 20, 445, 1), (32, 64, 148, 0)])
def test_threads_per_sm_of_an_fp32_gather(helper, width, source, blocks, many):
    """More threads, with fewer registers each, only where 384 do not hold all blocks at once, and not for narrow sources, whose loop is bound elsewhere."""
    assert helper.f32_many_blocks(width, source, C.c_longlong(blocks)) == many
