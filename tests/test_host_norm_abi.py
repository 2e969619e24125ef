"""The backward entry point of convolution + GroupNorm + ReLU checks its handle's device and, before that, every argument that it and the passes
behind it need: its first launch overwrites outputs.  The entry points that take the gradient of a
convolution's output refuse a null one (only the joint form works from rows that are packed already).  Needs no GPU; see test_host_abi."""
import ctypes as C

from test_host_abi import helper, i, lib, n, p  # noqa: F401  (fixtures and made-up arguments)
import pytest
import torch


@pytest.mark.skipif(torch.cuda.is_available(), reason="the calls would reach kernels with made-up pointers")
def test_conv_norm_checks_the_device(lib):  # noqa: F811
    l, h = lib
    rc = l.aprnet_conv333_norm_backward(h, i(0), i(8), i(8), i(1), p, p, C.c_int64(1 << 40), i(8), p, p, p, p, i(1), p, p, p, n, p, p, n, p, p, p, p, p, None)
    assert rc != 0 and b"device" in l.aprnet_last_error()


@pytest.mark.parametrize("name,args", [
    ("aprnet_conv333_rows_backward", (i(0), i(1), i(8), i(8), i(1), p, None, n, p, p, n, p, i(0), p, n, i(1), p, p, None)),
    ("aprnet_conv333_backward_tc_rows", (i(0), i(8), i(8), i(1), p, None, n, p, p, n, p, p, n, p, p, None)),
    ("aprnet_conv333_backward_tc_rows_pretree", (i(0), i(8), i(8), i(1), p, None, n, p, p, n, p, p, n, p, p, None))])
def test_null_gradients_are_refused(lib, name, args):  # noqa: F811
    l, h = lib
    rc = getattr(l, name)(h, *args)
    assert rc != 0 and b"bad argument" in l.aprnet_last_error()


# apr, level delta, cin, cout, slots, rows, conv_out, n, groups, gamma, beta, mean, rstd, relu, grad_y, weights, grad_input, ld_in, grad_weights,
# grad_tree, ld_tree, grad_gamma, grad_beta, partial, workspace, norm_workspace, stream
NORM = [None, i(0), i(8), i(8), i(1), p, p, n, i(8), p, p, p, p, i(1), p, p, p, n, p, p, n, p, p, p, p, p, None]
SMALL, ODD = C.c_int64(1), C.c_void_p(0x1008)          # the handle has 16 locations and 2 tree nodes


@pytest.mark.skipif(torch.cuda.is_available(), reason="a missing check would launch kernels on made-up pointers")
@pytest.mark.parametrize("at,value,message", [(k, None, b"bad argument") for k in (5, 6, 11, 12, 14, 15, 18, 19, 21, 22, 23, 24, 25)] +
                         [(4, i(0), b"bad argument"), (8, i(0), b"bad argument"), (8, i(3), b"bad argument"), (2, i(4), b"bad argument"),
                          (7, SMALL, b"leading dimension"), (17, SMALL, b"leading dimension"), (20, SMALL, b"leading dimension"),
                          (5, ODD, b"aligned"), (24, ODD, b"aligned")])
def test_conv_norm_checks_its_arguments_first(lib, at, value, message):  # noqa: F811
    l, h = lib
    args = [h] + NORM[1:]
    args[at] = value
    assert l.aprnet_conv333_norm_backward(*args) == -1 and message in l.aprnet_last_error()


@pytest.mark.skipif(torch.cuda.is_available(), reason="a missing check would launch kernels on made-up pointers")
def test_conv_norm_refuses_what_the_edge_plan_cannot_number(helper, lib):  # noqa: F811
    l, h = lib
    args = [h] + NORM[1:]
    args[7] = args[17] = args[20] = C.c_int64(1 << 40)
    for particles, rc, message in ((79536431, -2, b"device"), (79536432, -3, b"79.5 M"), (90000000, -3, b"79.5 M")):
        helper.set_particles(h, C.c_longlong(particles))
        try:
            assert l.aprnet_conv333_norm_backward(*args) == rc and message in l.aprnet_last_error()
        finally:
            helper.set_particles(h, C.c_longlong(16))
