"""Fused GroupNorm + ReLU for (batch, channels, particles) feature tensors.

Not part of the reference's `aprnet` API: its network blocks apply `torch.nn.GroupNorm` and `nn.ReLU`
after every convolution (apr_models/apr_models/unet/unet_parts.py:18-26).  `GroupNormReLU` computes the
same function (parameters `weight` / `bias` like `nn.GroupNorm`, so state dicts interchange) with
kernels sized for tens of millions of particles per row; the ReLU mask is recomputed in the backward
pass, so only the input and the per-group statistics are kept for it.
"""
import torch
from torch import nn
from torch.autograd import Function

from torch.nn.modules import module as _module

from _pyaprwrapper.aprnet.cuda import (conv333_forward_keep_rows, conv333_norm_backward, get_conv_precision, groupnorm_relu_backward,
                                       groupnorm_relu_forward, restrict_kernel333_backward, restrict_kernel333_forward)
from _pyaprwrapper.data_containers import APRPtrVector

from .conv import APRConv, Conv333Function


class GroupNormReLUFunction(Function):
    @staticmethod
    def forward(ctx, x, weight, bias, groups, eps, relu):
        x = x.contiguous()
        y, mean, rstd = groupnorm_relu_forward(x, weight, bias, groups, eps, relu)
        ctx.save_for_backward(x, weight, bias, mean, rstd)
        ctx.groups, ctx.relu = groups, relu
        return y

    @staticmethod
    def backward(ctx, grad_y):
        x, weight, bias, mean, rstd = ctx.saved_tensors
        dx, dgamma, dbeta = groupnorm_relu_backward(x, grad_y.contiguous(), weight, bias, mean, rstd, ctx.groups, ctx.relu)
        return dx, (dgamma if weight is not None else None), (dbeta if bias is not None else None), None, None, None


class GroupNormReLU(nn.Module):
    def __init__(self, num_groups, num_channels, eps=1e-5, affine=True, relu=True):
        super().__init__()
        assert num_channels % num_groups == 0
        self.num_groups, self.num_channels, self.eps, self.relu = num_groups, num_channels, eps, relu
        self.weight = nn.Parameter(torch.ones(num_channels)) if affine else None
        self.bias = nn.Parameter(torch.zeros(num_channels)) if affine else None

    def extra_repr(self):
        return '{}, {}, eps={}, relu={}'.format(self.num_groups, self.num_channels, self.eps, self.relu)

    def forward(self, x):
        return GroupNormReLUFunction.apply(x, self.weight, self.bias, self.num_groups, self.eps, self.relu)


class ConvGroupNormReLUFunction(Function):
    """3x3x3 convolution without a bias, GroupNorm and ReLU for one batch item in bf16 arithmetic.  The forward pass is that of the two
    functions; in the backward pass the gradient between them exists only as the packed bf16 rows that the convolution works from, written
    by the normalisation (same values, 8 of 18 bytes less per value)."""

    @staticmethod
    def forward(ctx, inputs, weights, gamma, beta, aprs, level_deltas, groups, eps, relu):
        num_levels = max(a.level_max() - a.level_min() + 1 for a in aprs)
        expanded = restrict_kernel333_forward(weights, num_levels)
        out, rows = conv333_forward_keep_rows(APRPtrVector(aprs), inputs, expanded, level_deltas, "bf16", None, True)
        y, mean, rstd = groupnorm_relu_forward(out, gamma, beta, groups, eps, relu)
        ctx.save_for_backward(expanded, level_deltas.clone(), rows, out, gamma, beta, mean, rstd)
        ctx.aprs, ctx.num_stencils, ctx.groups, ctx.relu = aprs, weights.shape[0], groups, relu
        return y

    @staticmethod
    def backward(ctx, grad_y):
        expanded, level_deltas, rows, out, gamma, beta, mean, rstd = ctx.saved_tensors
        grad_input, grad_expanded, dgamma, dbeta = conv333_norm_backward(APRPtrVector(ctx.aprs), rows, expanded, out, grad_y.contiguous(), gamma, beta, mean, rstd,
                                                                         ctx.groups, ctx.relu, level_deltas, bool(ctx.needs_input_grad[0]))
        return (grad_input, restrict_kernel333_backward(grad_expanded, ctx.num_stencils), dgamma if gamma is not None else None,
                dbeta if beta is not None else None, None, None, None, None, None)


def _plain(m, kind):
    """`m` is a module of exactly this kind that nothing observes: calling it is calling its `forward`."""
    return (type(m) is kind and "forward" not in m.__dict__ and
            not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or
                 _module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks or _module._global_backward_pre_hooks))


def conv_norm(conv, norm, x, aprs, level_deltas):
    """`norm(conv(x, aprs, level_deltas))` for an `APRConv` followed by a `GroupNormReLU`, as one function where both are plain modules and a
    backward pass of the convolution in bf16 arithmetic over one batch item can follow; as two calls otherwise, also where only the
    normalisation wants gradients: the convolution then keeps nothing and has no backward pass.  (More than four input channels: the weight gradient
    of a first layer reads the gradient channel by channel; up to 79.5 M locations: beyond them the input gradient does.)"""
    if (_plain(conv, APRConv) and _plain(norm, GroupNormReLU) and conv._function is Conv333Function and conv.bias is None and x.is_cuda and x.dim() == 3 and
            x.shape[0] == 1 and len(aprs) == 1 and 4 < x.shape[1] == conv.in_channels and norm.num_channels == conv.out_channels and
            27 * x.shape[2] + 1 < 2 ** 31 and (conv.precision or get_conv_precision()) == "bf16" and torch.is_grad_enabled()):
        tensors = [t for t in (x, conv.weight, norm.weight, norm.bias) if t is not None]
        if (x.requires_grad or conv.weight.requires_grad) and all(t.dtype == torch.float32 and t.device == x.device for t in tensors):
            return ConvGroupNormReLUFunction.apply(x, conv.weight, norm.weight, norm.bias, aprs, level_deltas, norm.num_groups, norm.eps, norm.relu)
    return norm(conv(x, aprs, level_deltas))
