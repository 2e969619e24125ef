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

from _pyaprwrapper.aprnet.cuda import (conv333_norm_backward, conv333_norm_forward, get_conv_precision, groupnorm_relu_backward,
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
    """3x3x3 convolution without a bias, GroupNorm and ReLU on float32 tensors.  The forward pass is that of the two functions, over `inputs` or the
    concatenation of `inputs` and `inputs1` along the channels, which is not written out.  keep (one batch item, bf16 arithmetic): a backward pass can follow, in which
    the gradient between the two exists only as the packed bf16 rows that the convolution works from, written by the normalisation (same values, 8 of
    18 bytes less per value).  Without it nothing is kept, and the entries behind the particles of a shorter item are not written between the two."""

    @staticmethod
    def forward(ctx, inputs, inputs1, weights, gamma, beta, aprs, level_deltas, groups, eps, relu, precision, keep):
        num_levels = max(a.level_max() - a.level_min() + 1 for a in aprs)
        expanded = restrict_kernel333_forward(weights, num_levels)
        y, *kept = conv333_norm_forward(APRPtrVector(aprs), inputs, inputs1, expanded, level_deltas, precision, gamma, beta, groups, eps, relu, keep)
        if keep:
            mean, rstd, out, rows = kept
            ctx.save_for_backward(expanded, level_deltas.clone(), rows, out, gamma, beta, mean, rstd)
            ctx.aprs, ctx.num_stencils, ctx.groups, ctx.relu, ctx.split = aprs, weights.shape[0], groups, relu, inputs.shape[1]
        return y

    @staticmethod
    def backward(ctx, grad_y):
        expanded, level_deltas, rows, out, gamma, beta, mean, rstd = ctx.saved_tensors
        wanted = ctx.needs_input_grad
        grad_input, grad_expanded, dgamma, dbeta = conv333_norm_backward(APRPtrVector(ctx.aprs), rows, expanded, out, grad_y.contiguous(), gamma, beta, mean, rstd,
                                                                         ctx.groups, ctx.relu, level_deltas, bool(wanted[0] or wanted[1]))
        # two inputs: each has its channels of one gradient
        grad_input0 = grad_input if not wanted[0] or ctx.split == expanded.shape[2] else grad_input[:, :ctx.split]
        return (grad_input0 if wanted[0] else None, grad_input[:, ctx.split:] if wanted[1] else None, restrict_kernel333_backward(grad_expanded, ctx.num_stencils),
                dgamma if gamma is not None else None, dbeta if beta is not None else None, None, None, None, None, None, None, None)


def _plain(m, kind):
    """`m` is a module of exactly this kind that nothing observes: calling it is calling its `forward`."""
    return (type(m) is kind and "forward" not in m.__dict__ and
            not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or
                 _module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks or _module._global_backward_pre_hooks))


def _backward_follows(conv, norm, x, skip, aprs):
    """Whether the convolution and the normalisation are one function: None if not, else whether a backward pass can follow.  (What refuses most calls comes first: with all
    checks made for every call, small layers that end in two calls took 7 us more.)"""
    if type(conv) is not APRConv or type(norm) is not GroupNormReLU or conv.bias is not None:
        return None
    weight, gamma, beta = conv.weight, norm.weight, norm.bias
    features = x.requires_grad or weight.requires_grad or (skip is not None and skip.requires_grad)
    wanted = (features or (gamma is not None and gamma.requires_grad) or (beta is not None and beta.requires_grad)) and torch.is_grad_enabled()
    if wanted and not (features and conv.in_channels > 4 and len(aprs) == 1 and (conv.precision or get_conv_precision()) == "bf16"):
        return None
    if not (x.is_cuda and x.dim() == 3 and x.is_contiguous() and _plain(conv, APRConv) and _plain(norm, GroupNormReLU) and conv._function is Conv333Function):
        return None
    batch, channels, n = x.shape
    if (batch != len(aprs) or batch == 0 or channels + (0 if skip is None else skip.shape[1]) != conv.in_channels or norm.num_channels != conv.out_channels or
            (wanted and 27 * n + 1 >= 2 ** 31)):
        return None
    for t in (x, weight, gamma, beta):
        if t is not None and (t.dtype is not torch.float32 or t.device != x.device):
            return None
    return wanted


def _two_inputs(conv, skip, x):
    """The kernels take the two tensors as they are: more than four channels together, the first tensor's a multiple of four."""
    return (conv.in_channels > 4 and skip.dim() == x.dim() == 3 and skip.shape[1] % 4 == 0 and skip.shape[1] > 0 and x.shape[1] > 0 and
            skip.shape[0] == x.shape[0] and skip.shape[2] == x.shape[2] and skip.dtype == x.dtype and skip.device == x.device and skip.is_contiguous() and x.is_contiguous())


def conv_norm(conv, norm, x, aprs, level_deltas, skip=None):
    """`norm(conv(x, aprs, level_deltas))` for an `APRConv` followed by a `GroupNormReLU`; with `skip`, x is `torch.cat([skip, x], 1)`, which is written out where the
    kernels do not take the two tensors.  One function where both are plain modules and either no gradient is wanted or a backward pass of the convolution in bf16
    arithmetic over one batch item can follow; two calls otherwise, also where only the normalisation wants gradients: the convolution then keeps nothing and has no backward pass.
    (More than four input channels in a backward pass: the weight gradient of a first layer reads the gradient channel by channel; up to 79.5 M
    locations: beyond them the input gradient does.)"""
    if skip is not None and not (type(conv) is APRConv and _two_inputs(conv, skip, x)):
        x, skip = torch.cat([skip, x], dim=1), None
    wanted = _backward_follows(conv, norm, x, skip, aprs)
    if wanted is not None:
        return ConvGroupNormReLUFunction.apply(x if skip is None else skip, None if skip is None else x, conv.weight, norm.weight, norm.bias, aprs, level_deltas,
                                               norm.num_groups, norm.eps, norm.relu, conv.precision or get_conv_precision(), wanted)
    if skip is not None:
        x = torch.cat([skip, x], dim=1)
    return norm(conv(x, aprs, level_deltas))
