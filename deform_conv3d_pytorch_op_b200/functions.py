"""autograd Functions with the reference's call signatures.

* :class:`ConvOffset3dFunction` -- deform3d/deform_conv3d_functions/deform_conv3d_function.py:7-77
* :class:`ConvOffset2dFunction` -- deform2d_double/deform_conv2d_functions/deform_conv2d_function.py:7-77
* :class:`Conv2dFunction`       -- conv2d/conv2d_functions/conv2d_function.py:8-67
* :class:`Conv3dFunction`       -- the same call form over three spatial axes (no counterpart in the reference)
* :class:`DeformLayerFunction`  -- offset-producing convolution + deformable convolution as one unit, the
  caller pattern of deform3d/test_model.py:18-30
* :class:`LegacyConvOffset2dFunction` -- the stateful fp32 2-D form,
  deform2d/deform_conv2d_functions/deform_conv2d_function.py:7-57

``.apply`` keeps the reference's positional order and its gradients the same slots.  Differences:
gradients are computed only for the inputs that need them (the reference always computes dX and dOffset
together), and two optional trailing arguments select the arithmetic (``precision``: exact | bf16 | auto)
and the 3-D out-of-bounds offset pseudo-gradient (``oob_offset_grad``).

The work behind ``.apply`` -- checks, allocation, the library call, the graph node of the backward pass -- is C++
(``csrc/dcn_torch.cpp``): in Python it cost more than the kernels of a small layer.  The classes are therefore no
subclasses of ``torch.autograd.Function``; where a trace, a function transform (``torch.func``) or a forward-mode
derivative needs one, the call goes through the ``_...Function`` of the same arguments below.
"""
from __future__ import annotations

from torch.autograd import Function
from torch.autograd.function import once_differentiable

from . import _lib
from .ops import Op, check_status, status_check_enabled


def _tup(v, n):
    return tuple(v) if isinstance(v, (tuple, list)) else (v,) * n


def _check(x):
    if status_check_enabled():
        check_status(x.device)


class _DeformFunction(Function):
    @staticmethod
    def forward(ctx, ndim, inputs, offset, weight, bias=None, stride=1, padding=0, dilation=1, channel_per_group=1,
                group=1, precision=None, oob_offset_grad=None):
        if inputs.dim() != ndim + 2:
            raise RuntimeError("input dim")
        ctx.op = Op(inputs, weight, _tup(stride, ndim), _tup(padding, ndim), _tup(dilation, ndim), channel_per_group,
                    group, oob_offset_grad=oob_offset_grad, precision=precision)
        ctx.save_for_backward(inputs, offset, weight)
        return ctx.op.forward(inputs, offset, weight, bias)

    @staticmethod
    @once_differentiable
    def backward(ctx, dy):
        grads = ctx.op.backward(*ctx.saved_tensors, dy, *ctx.needs_input_grad[1:5])
        _check(dy)
        return (None,) + grads + (None,) * 7


class _PlainFunction(Function):
    @staticmethod
    def forward(ctx, ndim, inputs, weight, bias=None, stride=1, padding=0, dilation=1, group=1, precision=None):
        if inputs.dim() != ndim + 2:
            raise RuntimeError("input dim")
        ctx.op = Op(inputs, weight, _tup(stride, ndim), _tup(padding, ndim), _tup(dilation, ndim), inputs.size(1),
                    group, deformable=False, std_size_rule=True, precision=precision)
        ctx.save_for_backward(inputs, weight)
        return ctx.op.forward(inputs, None, weight, bias)

    @staticmethod
    @once_differentiable
    def backward(ctx, dy):
        inputs, weight = ctx.saved_tensors
        _, need_x, need_w, need_b = ctx.needs_input_grad[:4]
        dx, _, dw, db = ctx.op.backward(inputs, None, weight, dy, need_x, False, need_w, need_b)
        return (None, dx, dw, db) + (None,) * 5


class _LayerFunction(Function):
    @staticmethod
    def forward(ctx, inputs, offset_weight, offset_bias, weight, bias, stride, padding, dilation, channel_per_group=1,
                group=1, precision=None, oob_offset_grad=None):
        ndim = inputs.dim() - 2
        ctx.op = Op(inputs, weight, _tup(stride, ndim), _tup(padding, ndim), _tup(dilation, ndim), channel_per_group,
                    group, oob_offset_grad=oob_offset_grad, precision=precision)
        y, offset = ctx.op.layer_forward(inputs, offset_weight, offset_bias, weight, bias)
        ctx.save_for_backward(inputs, offset, offset_weight, weight)
        return y

    @staticmethod
    @once_differentiable
    def backward(ctx, dy):
        grads = ctx.op.layer_backward(*ctx.saved_tensors, dy, *ctx.needs_input_grad[:5])
        _check(dy)
        return grads + (None,) * 7


class ConvOffset3dFunction:
    """``apply(inputs, offset, weight, bias=None, stride=(1, 1, 1), padding=(0, 0, 0), dilation=(1, 1, 1),
    channel_per_group=1, group=1, precision=None, oob_offset_grad=None)``"""

    @staticmethod
    def apply(*args):
        y = _lib.native().conv_offset3d(*args)
        return _DeformFunction.apply(3, *args) if y is NotImplemented else y


class ConvOffset2dFunction:
    """``apply(inputs, offset, weight, bias=None, stride=(1, 1), padding=(0, 0), dilation=(1, 1),
    channel_per_group=1, group=1, precision=None, oob_offset_grad=None)``"""

    @staticmethod
    def apply(*args):
        y = _lib.native().conv_offset2d(*args)
        return _DeformFunction.apply(2, *args) if y is NotImplemented else y


class Conv2dFunction:
    """Plain (integer-tap) convolution on the same kernels with the deformable part switched off:
    ``apply(inputs, weight, bias=None, stride=(1, 1), padding=(0, 0), dilation=(1, 1), group=1, precision=None)``"""

    @staticmethod
    def apply(*args):
        y = _lib.native().conv2d(*args)
        return _PlainFunction.apply(2, *args) if y is NotImplemented else y


class Conv3dFunction:
    """The 3-D counterpart of :class:`Conv2dFunction` (the reference's plain-convolution package is 2-D only,
    conv2d/lib/conv2d_cuda.cpp:77-290; the same im2col + GEMM structure over (l, h, w))."""

    @staticmethod
    def apply(*args):
        y = _lib.native().conv3d(*args)
        return _PlainFunction.apply(3, *args) if y is NotImplemented else y


class DeformLayerFunction:
    """``apply(inputs, offset_weight, offset_bias, weight, bias, stride, padding, dilation, channel_per_group=1,
    group=1[, precision, oob_offset_grad])``: the offset-producing convolution and the deformable convolution of the
    reference's model scripts (deform3d/test_model.py:18-30, deform2d/test_model.py:19-31) as one differentiable
    unit; 2-D or 3-D by the input's rank.  The offsets never pass through the caller."""

    @staticmethod
    def apply(*args):
        y = _lib.native().deform_layer(*args)
        return _LayerFunction.apply(*args) if y is NotImplemented else y


class LegacyConvOffset2dFunction:
    """``ConvOffset2dFunction(stride, padding, channel_per_group)(input, offset, weight)`` -- the stateful call
    form of the fp32 2-D package (no dilation, no groups, no bias)."""

    def __init__(self, stride, padding, channel_per_group):
        self.stride = _tup(stride, 2)
        self.padding = _tup(padding, 2)
        self.channel_per_group = channel_per_group

    def __call__(self, inputs, offset, weight):
        return ConvOffset2dFunction.apply(inputs, offset, weight, None, self.stride, self.padding, (1, 1),
                                          self.channel_per_group, 1)
