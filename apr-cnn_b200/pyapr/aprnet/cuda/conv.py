"""`APRConv` with 3x3x3 and 1x1x1 stencils (reference: pyapr/aprnet/cuda/conv.py:12-94).

Same constructor, parameter shapes (`weight`: (nstencils, out, in, k, k, k), `bias`: (out,)),
initialisation and forward signature `(features, aprs, level_deltas)` as the reference module, so
checkpoints and calling code interchange.
"""
import math

import torch
from torch import nn
from torch.autograd import Function
from torch.nn import init

from _pyaprwrapper.data_containers import APRPtrVector
from _pyaprwrapper.aprnet.cuda import (conv111_backward, conv111_backward_with_bias, conv111_forward, conv333_backward_with_rows,
                                       conv333_backward_with_rows_bias, conv333_backward_with_tree,
                                       conv333_forward_keep_rows, conv333_forward_keep_tree, get_conv_precision,
                                       restrict_kernel333_backward, restrict_kernel333_forward)


def _kernel_bias(bias, inputs, weights):
    """The bias as the kernels add it (contiguous, one value per output channel, the features' type and device); None where torch has
    to add it afterwards by its own rules (another type, a broadcast value) or there is none."""
    if bias is None or bias.dtype != inputs.dtype or bias.device != inputs.device or bias.numel() != weights.shape[1]:
        return None
    return bias.contiguous()


class Conv333Function(Function):
    """3x3x3 stencil: the given stencils are expanded to one per level, then applied per level."""

    @staticmethod
    def forward(ctx, inputs, weights, bias, aprs, level_deltas, precision=None, keep=True):
        # keep: something for a backward pass is kept (False where no gradient can be wanted: one item's scratch instead of the
        # packed rows of the whole batch)
        num_levels = max(a.level_max() - a.level_min() + 1 for a in aprs)
        expanded = restrict_kernel333_forward(weights, num_levels)
        ctx.aprs = aprs
        ctx.num_stencils = weights.shape[0]
        # float32: the backward pass works from the packed rows of the input (particles + tree means, bf16 or fp32 as the
        # layer's arithmetic wants them) that the forward pass produced anyway; they replace the input among the saved
        # tensors and spare the backward pass the tree fill and the packing.  The bias is added where the output is written.
        ctx.packed = inputs.dtype == torch.float32
        if ctx.packed:
            ctx.precision = precision or get_conv_precision()
            fused = _kernel_bias(bias, inputs, weights)
            out, rows = conv333_forward_keep_rows(APRPtrVector(aprs), inputs, expanded, level_deltas, ctx.precision, fused, keep)
            if keep:
                ctx.save_for_backward(expanded, bias, level_deltas.clone(), rows)
            return out if bias is None or fused is not None else out + bias.view(1, -1, 1)
        # float64: the tree means computed by the forward pass are kept (1/7 of the input's size) so that the
        # backward pass does not have to fill the tree again
        out, tree = conv333_forward_keep_tree(APRPtrVector(aprs), inputs, expanded, level_deltas)
        ctx.save_for_backward(inputs, expanded, bias, level_deltas.clone(), tree)
        if bias is not None:
            out = out + bias.view(1, -1, 1)
        return out

    @staticmethod
    def backward(ctx, grad_output):
        grad_output = grad_output.contiguous()
        if ctx.packed:
            expanded, bias, level_deltas, rows = ctx.saved_tensors
            backward = conv333_backward_with_rows if bias is None else conv333_backward_with_rows_bias
            grad_input, grad_expanded, *grad_bias = backward(APRPtrVector(ctx.aprs), rows, expanded, grad_output, level_deltas, bool(ctx.needs_input_grad[0]), ctx.precision)
            grad_weights = restrict_kernel333_backward(grad_expanded, ctx.num_stencils)
            return grad_input, grad_weights, grad_bias[0] if grad_bias else None, None, None, None, None
        inputs, expanded, bias, level_deltas, tree = ctx.saved_tensors
        grad_input, grad_expanded = conv333_backward_with_tree(APRPtrVector(ctx.aprs), inputs, expanded, grad_output, level_deltas, tree)
        grad_weights = restrict_kernel333_backward(grad_expanded, ctx.num_stencils)
        grad_bias = grad_output.sum(dim=(0, 2)) if bias is not None else None
        return grad_input, grad_weights, grad_bias, None, None, None, None


class Conv111Function(Function):
    """1x1x1 stencil: a per-level channel mix, no neighbour access and no stencil expansion."""

    @staticmethod
    def forward(ctx, inputs, weights, bias, aprs, level_deltas, precision=None):
        ctx.aprs = aprs
        ctx.precision = precision or ""
        ctx.save_for_backward(inputs, weights, bias, level_deltas.clone())
        fused = _kernel_bias(bias, inputs, weights)
        out = conv111_forward(APRPtrVector(aprs), inputs, weights, level_deltas, ctx.precision, fused)
        return out if bias is None or fused is not None else out + bias.view(1, -1, 1)

    @staticmethod
    def backward(ctx, grad_output):
        inputs, weights, bias, level_deltas = ctx.saved_tensors
        grad_output = grad_output.contiguous()
        backward = conv111_backward if bias is None else conv111_backward_with_bias
        grad_input, grad_weights, *grad_bias = backward(APRPtrVector(ctx.aprs), inputs, weights, grad_output, level_deltas, ctx.precision)
        return grad_input, grad_weights, grad_bias[0] if grad_bias else None, None, None, None


_FUNCTIONS = {(1, 1, 1): Conv111Function, (3, 3, 3): Conv333Function}


class APRConv(nn.Module):
    """`precision` (not in the reference): arithmetic of the layer on float32 tensors, "fp32" (CUDA-core kernels,
    exact) or "bf16" (tensor cores, bf16 operands with fp32 accumulation); None follows the process-wide setting
    (`set_conv_precision`)."""

    def __init__(self, in_channels, out_channels, nstencils=1, kernel_size=(3, 3, 3), bias=True, precision=None):
        super().__init__()
        assert precision in (None, "fp32", "bf16")
        self.precision = precision
        kernel_size = tuple(kernel_size)
        assert kernel_size in _FUNCTIONS, \
            'aprnet.cuda.APRConv currently only supports kernels of size (1, 1, 1) and (3, 3, 3)'
        self._function = _FUNCTIONS[kernel_size]
        self.in_channels = in_channels
        self.out_channels = out_channels
        self.nstencils = nstencils
        self.kernel_size = kernel_size
        self.weight = nn.Parameter(torch.empty(nstencils, out_channels, in_channels, *kernel_size))
        self.bias = nn.Parameter(torch.empty(out_channels)) if bias else None
        self.reset_parameters()

    def extra_repr(self):
        return '{}, {}, kernel_size={}, nstencils={}, bias={}'.format(
            self.in_channels, self.out_channels, self.kernel_size, self.nstencils, self.bias is not None)

    def reset_parameters(self):
        init.kaiming_uniform_(self.weight, a=math.sqrt(5))
        if self.bias is not None:
            fan_in, _ = init._calculate_fan_in_and_fan_out(self.weight)
            bound = 1 / math.sqrt(fan_in)
            init.uniform_(self.bias, -bound, bound)

    def forward(self, input_features, aprs, level_deltas):
        if self._function is Conv111Function:
            return Conv111Function.apply(input_features, self.weight, self.bias, aprs, level_deltas, self.precision)
        keep = torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (input_features, self.weight, self.bias))
        return Conv333Function.apply(input_features, self.weight, self.bias, aprs, level_deltas, self.precision, keep)
