"""The backward entry point of convolution + GroupNorm + ReLU checks its handle's device, and the entry points that take the gradient of a
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
