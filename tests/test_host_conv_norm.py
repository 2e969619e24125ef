"""`conv_norm` settles what refuses most calls before it looks at the tensors: small layers that end in two calls are bound by the host."""
import pytest
import torch

from pyapr.aprnet import cuda as ops


class Features:
    """Stands for a tensor of which only `requires_grad` may be asked."""
    requires_grad = True

    def __getattr__(self, name):
        raise AssertionError("looked at " + name)


@pytest.mark.parametrize("channels,precision,aprs,bias", [(8, "fp32", 1, False), (4, "bf16", 1, False), (8, "bf16", 2, False), (8, "bf16", 1, True)])
def test_refused_without_a_look_at_the_features(monkeypatch, channels, precision, aprs, bias):
    conv, norm = ops.APRConv(channels, 8, bias=bias, precision=precision), ops.GroupNormReLU(2, 8)
    monkeypatch.setattr(ops.APRConv, "forward", lambda self, x, a, ld: x)
    monkeypatch.setattr(ops.GroupNormReLU, "forward", lambda self, x: x)
    x = Features()
    with torch.enable_grad():
        assert ops.conv_norm(conv, norm, x, [None] * aprs, None) is x
