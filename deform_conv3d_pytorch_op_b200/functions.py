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
(``csrc/dcn_torch.cpp``): in Python it cost more than the kernels of a small layer.
"""
from __future__ import annotations

from . import _lib


def _tup(v, n):
    return tuple(v) if isinstance(v, (tuple, list)) else (v,) * n


class ConvOffset3dFunction:
    """``apply(inputs, offset, weight, bias=None, stride=(1, 1, 1), padding=(0, 0, 0), dilation=(1, 1, 1),
    channel_per_group=1, group=1, precision=None, oob_offset_grad=None)``"""

    @staticmethod
    def apply(*args):
        return _lib.native().conv_offset3d(*args)


class ConvOffset2dFunction:
    """``apply(inputs, offset, weight, bias=None, stride=(1, 1), padding=(0, 0), dilation=(1, 1),
    channel_per_group=1, group=1, precision=None, oob_offset_grad=None)``"""

    @staticmethod
    def apply(*args):
        return _lib.native().conv_offset2d(*args)


class Conv2dFunction:
    """Plain (integer-tap) convolution on the same kernels with the deformable part switched off:
    ``apply(inputs, weight, bias=None, stride=(1, 1), padding=(0, 0), dilation=(1, 1), group=1, precision=None)``"""

    @staticmethod
    def apply(*args):
        return _lib.native().conv2d(*args)


class Conv3dFunction:
    """The 3-D counterpart of :class:`Conv2dFunction` (the reference's plain-convolution package is 2-D only,
    conv2d/lib/conv2d_cuda.cpp:77-290; the same im2col + GEMM structure over (l, h, w))."""

    @staticmethod
    def apply(*args):
        return _lib.native().conv3d(*args)


class DeformLayerFunction:
    """``apply(inputs, offset_weight, offset_bias, weight, bias, stride, padding, dilation, channel_per_group=1,
    group=1[, precision, oob_offset_grad])``: the offset-producing convolution and the deformable convolution of the
    reference's model scripts (deform3d/test_model.py:18-30, deform2d/test_model.py:19-31) as one differentiable
    unit; 2-D or 3-D by the input's rank.  The offsets never pass through the caller."""

    @staticmethod
    def apply(*args):
        return _lib.native().deform_layer(*args)


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
