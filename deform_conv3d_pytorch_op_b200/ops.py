"""Tensor-level entry points over the C ABI: the three passes of the operator on torch CUDA tensors.

These are the counterparts of the reference's FFI calls (``deform_conv3d_op.deform_conv_forward_cuda`` and
siblings, deform3d/lib/deform_conv3d_cuda.h:12-34) with the output allocation the reference does in Python
(deform3d/deform_conv3d_functions/deform_conv3d_function.py:26-32, 53-54, 64) folded in.  torch is used for
device memory and the current stream only; all arithmetic happens in libdcn.so.
"""
from __future__ import annotations

import ctypes
import os
from typing import Optional, Tuple

import torch

from . import _lib
from ._lib import DcnError

def default_precision() -> str:
    """``DCN_PRECISION`` = exact | bf16 | auto (default exact: compute in the tensor dtype)."""
    return os.environ.get("DCN_PRECISION", "exact").lower()


def default_oob_offset_grad() -> bool:
    """``DCN_OOB_OFFSET_GRAD`` = reference | zero (default reference; only 3-D has the term)."""
    return os.environ.get("DCN_OOB_OFFSET_GRAD", "reference").lower() != "zero"


def check_status(device=None) -> None:
    """Reads and clears the library's device-side status word on ``device`` (default: the current CUDA device)
    and raises :class:`DcnError` if a bounded device-side wait of a tensor-core kernel gave up since the last
    check.  Synchronises the device's current stream.  The word is sticky and process-wide per device, so a check
    tells that *some* call since the previous check failed, not which one: check once per step (or per call while
    debugging; ``DCN_CHECK_STATUS=1`` makes every backward pass of the autograd Functions do so)."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(dev):
        _lib.check(_lib.lib().dcn_check_status(_lib.current_stream(dev)), "device status")


def status_check_enabled() -> bool:
    """Whether a backward pass checks the status word (``DCN_CHECK_STATUS=1``, and not while a stream is captured)."""
    return os.environ.get("DCN_CHECK_STATUS", "0") not in ("", "0") and not torch.cuda.is_current_stream_capturing()


def _nvtx_enabled() -> bool:
    """``DCN_NVTX=1``: wrap every library call of :class:`Op` in an NVTX range named after the entry point, so that
    the passes show up by name on a profiler's timeline (the reference has only wall-clock prints,
    deform2d/test_function.py:30-58)."""
    return os.environ.get("DCN_NVTX", "0") not in ("", "0")


class _Range:
    def __init__(self, name: str):
        self.on = _nvtx_enabled()
        self.name = name

    def __enter__(self):
        if self.on:
            torch.cuda.nvtx.range_push(self.name)

    def __exit__(self, *exc):
        if self.on:
            torch.cuda.nvtx.range_pop()
        return False


def _prep(t: Optional[torch.Tensor], name: str, ref: Optional[torch.Tensor] = None,
          memory_format: torch.memory_format = torch.contiguous_format) -> Optional[torch.Tensor]:
    if t is None:
        return None
    if not t.is_cuda:
        raise DcnError("%s must be a CUDA tensor (there is no CPU implementation)" % name)
    if ref is not None:
        if t.device != ref.device:
            raise DcnError("%s is on %s but input is on %s" % (name, t.device, ref.device))
        if t.dtype != ref.dtype:
            raise DcnError("%s has dtype %s but input has %s" % (name, t.dtype, ref.dtype))
    return t.contiguous(memory_format=memory_format)


class Op:
    """One validated operator instance (geometry + precision) bound to a device."""

    def __init__(self, x: torch.Tensor, weight: torch.Tensor, stride, padding, dilation, channel_per_group: int,
                 group: int, deformable: bool = True, std_size_rule: bool = False,
                 oob_offset_grad: Optional[bool] = None, precision: Optional[str] = None,
                 channels_last: Optional[bool] = None):
        # Checks, the `auto` rule and the storage order are those of the autograd Functions (csrc/dcn_torch.cpp).
        # (precision None: default_precision(); oob_offset_grad None: default_oob_offset_grad()).  Channels-last activations (torch.channels_last / channels_last_3d storage) are taken and produced as
        # they are by the bf16 path: no layout pass around the kernels.  Default: follow the input's memory format.
        p = _lib.dcn_problem.from_buffer_copy(_lib.native().problem(
            x, weight, *[v if isinstance(v, int) else tuple(int(a) for a in v) for v in (stride, padding, dilation)],
            int(channel_per_group), int(group), deformable, std_size_rule, oob_offset_grad, precision, channels_last))
        ndim = self.ndim = p.ndim
        self.device = x.device
        self.dtype = x.dtype
        cpg = p.cpg
        self.memory_format = torch.channels_last if ndim == 2 else torch.channels_last_3d
        self.p = p
        self.channels_last = bool(p.channels_last)
        self.deformable = deformable
        self.out_size = _lib.output_size(p)
        self.offset_channels = (x.size(1) // cpg) * int(torch.Size(weight.shape[2:]).numel()) * ndim
        self.N, self.C, self.O = x.size(0), x.size(1), weight.size(0)
        self.weight_shape = tuple(weight.shape)

    # -- helpers ---------------------------------------------------------------------------------
    def _act(self, t: Optional[torch.Tensor], name: str, ref: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
        """An activation-like tensor (input, output gradient) in the storage order the problem was built for."""
        return _prep(t, name, ref, self.memory_format if self.channels_last else torch.contiguous_format)

    def _new_act(self, shape, like: torch.Tensor, zero: bool = False) -> torch.Tensor:
        mf = self.memory_format if self.channels_last else torch.contiguous_format
        t = torch.empty(tuple(shape), dtype=like.dtype, device=like.device, memory_format=mf)
        return t.zero_() if zero else t

    def _scratch(self, nbytes: int, least: int = 0):
        """(workspace, its bytes).  The exact precision also runs without one, on slower kernels: it goes on with the
        ``least`` that a call cannot do without where the allocator has no room for ``nbytes``."""
        if nbytes == 0:
            return None, 0
        try:
            return torch.empty(nbytes, dtype=torch.uint8, device=self.device), nbytes
        except torch.OutOfMemoryError:
            if self.p.precision != _lib.PREC_EXACT or nbytes == least:
                raise
        return self._scratch(least, least)

    def _ws(self, which: int):
        return self._scratch(_lib.lib().dcn_workspace_bytes(ctypes.byref(self.p), which))

    def _check_offset(self, offset: torch.Tensor):
        want = (self.N, self.offset_channels) + tuple(self.out_size)
        if tuple(offset.shape) != want:
            raise DcnError("offset shape %s, expected %s" % (tuple(offset.shape), want))

    # -- passes ----------------------------------------------------------------------------------
    def backward(self, x, offset, weight, dy, want_dx=True, want_doffset=True, want_dw=True, want_dbias=False,
                 x_channels_last: Optional[torch.Tensor] = None):
        """All gradients through the fused entry point (outputs overwritten; scratch shared between the data
        and weight kernels).  ``x_channels_last``: the forward workspace kept by :meth:`forward` (bf16 path)."""
        x = self._act(x, "input")
        weight = _prep(weight, "weight", x)
        dy = self._act(dy, "grad_output", x)
        offset = _prep(offset, "offset", x) if self.deformable else None
        if not self.deformable:
            want_doffset = False
        dx = self._new_act(x.shape, x) if want_dx else None
        doff = torch.empty_like(offset) if want_doffset else None
        dw = torch.empty(self.weight_shape, dtype=x.dtype, device=x.device) if want_dw else None
        db = torch.empty(self.O, dtype=x.dtype, device=x.device) if want_dbias else None
        ws, nb = self._ws(_lib.PASS_BACKWARD)
        with torch.cuda.device(x.device), _Range("dcn_backward"):
            st = _lib.lib().dcn_backward(ctypes.byref(self.p), _lib.ptr(x), _lib.ptr(offset), _lib.ptr(weight),
                                         _lib.ptr(dy), _lib.ptr(x_channels_last), _lib.ptr(dx), _lib.ptr(doff),
                                         _lib.ptr(dw), _lib.ptr(db), _lib.ptr(ws), nb, _lib.current_stream(x.device))
        _lib.check(st, "dcn_backward")
        return dx, doff, dw, db

    def forward(self, x, offset, weight, bias=None, keep_workspace: bool = False):
        x = self._act(x, "input")
        weight = _prep(weight, "weight", x)
        bias = _prep(bias, "bias", x)
        if self.deformable:
            offset = _prep(offset, "offset", x)
            self._check_offset(offset)
        else:
            offset = None
        y = self._new_act((self.N, self.O) + tuple(self.out_size), x)
        ws, nb = self._ws(_lib.PASS_FORWARD)
        with torch.cuda.device(x.device), _Range("dcn_forward"):
            st = _lib.lib().dcn_forward(ctypes.byref(self.p), _lib.ptr(x), _lib.ptr(offset), _lib.ptr(weight),
                                        _lib.ptr(bias), _lib.ptr(y), _lib.ptr(ws), nb, _lib.current_stream(x.device))
        _lib.check(st, "dcn_forward")
        if keep_workspace:
            # the channels-last bf16 copy of x sits at the start of the workspace; backward can take it over
            return y, ws
        return y

    def backward_data(self, x, offset, weight, dy, want_dx=True, want_doffset=True
                      ) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
        weight = _prep(weight, "weight")
        dy = self._act(dy, "grad_output", weight)
        dx = doff = None
        if self.deformable:
            x = self._act(x, "input", weight)
            offset = _prep(offset, "offset", weight)
            self._check_offset(offset)
        else:
            offset = None
            want_doffset = False
        if want_dx:
            dx = self._new_act((self.N, self.C) + tuple(self.p.in_)[3 - self.ndim:], dy, zero=True)
        if want_doffset:
            doff = torch.empty((self.N, self.offset_channels) + tuple(self.out_size), dtype=dy.dtype, device=dy.device)
        if dx is None and doff is None:
            return None, None
        ws, nb = self._ws(_lib.PASS_BACKWARD_DATA)
        with torch.cuda.device(dy.device), _Range("dcn_backward_data"):
            st = _lib.lib().dcn_backward_data(ctypes.byref(self.p), _lib.ptr(x) if self.deformable else None,
                                              _lib.ptr(offset), _lib.ptr(weight), _lib.ptr(dy), _lib.ptr(dx),
                                              _lib.ptr(doff), _lib.ptr(ws), nb, _lib.current_stream(dy.device))
        _lib.check(st, "dcn_backward_data")
        return dx, doff

    def backward_weight(self, x, offset, dy, want_dw=True, want_dbias=False
                        ) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
        x = self._act(x, "input")
        dy = self._act(dy, "grad_output", x)
        offset = _prep(offset, "offset", x) if self.deformable else None
        dw = torch.zeros(self.weight_shape, dtype=x.dtype, device=x.device) if want_dw else None
        db = torch.empty(self.O, dtype=x.dtype, device=x.device) if want_dbias else None
        if dw is None and db is None:
            return None, None
        ws, nb = self._ws(_lib.PASS_BACKWARD_WEIGHT) if want_dw else (None, 0)
        with torch.cuda.device(x.device), _Range("dcn_backward_weight"):
            st = _lib.lib().dcn_backward_weight(ctypes.byref(self.p), _lib.ptr(x), _lib.ptr(offset), _lib.ptr(dy),
                                                _lib.ptr(dw), _lib.ptr(db), _lib.ptr(ws), nb,
                                                _lib.current_stream(x.device))
        _lib.check(st, "dcn_backward_weight")
        return dw, db

    # -- deformable layer: offset-producing convolution + deformable convolution in one call -------------------
    def offset_weight_shape(self):
        """Weight shape of the convolution that produces this operator's offsets: [dg*kv*D, C, k...]."""
        return (self.offset_channels, self.C) + tuple(self.weight_shape[2:])

    def _layer_ws(self, which: int):
        nbytes = _lib.lib().dcn_layer_workspace_bytes(ctypes.byref(self.p), which)
        doff = self.N * self.offset_channels * int(torch.Size(self.out_size).numel()) * (8 if self.p.dtype else 4)
        return self._scratch(nbytes, (doff + 255) // 256 * 256 if which == _lib.PASS_BACKWARD else 0)

    def layer_forward(self, x, offset_weight, offset_bias, weight, bias=None, keep_workspace: bool = False):
        """offset = conv(x, offset_weight) + offset_bias; y = deform_conv(x, offset, weight) + bias.
        Returns (y, offset[, workspace])."""
        if not self.deformable:
            raise DcnError("the layer entry points need a deformable operator")
        x = self._act(x, "input")
        weight = _prep(weight, "weight", x)
        bias = _prep(bias, "bias", x)
        offset_weight = _prep(offset_weight, "offset_weight", x)
        offset_bias = _prep(offset_bias, "offset_bias", x)
        if tuple(offset_weight.shape) != self.offset_weight_shape():
            raise DcnError("offset_weight shape %s, expected %s" % (tuple(offset_weight.shape),
                                                                    self.offset_weight_shape()))
        y = self._new_act((self.N, self.O) + tuple(self.out_size), x)
        offset = torch.empty((self.N, self.offset_channels) + tuple(self.out_size), dtype=x.dtype, device=x.device)
        ws, nb = self._layer_ws(_lib.PASS_FORWARD)
        with torch.cuda.device(x.device), _Range("dcn_layer_forward"):
            st = _lib.lib().dcn_layer_forward(ctypes.byref(self.p), _lib.ptr(x), _lib.ptr(offset_weight),
                                              _lib.ptr(offset_bias), _lib.ptr(weight), _lib.ptr(bias), _lib.ptr(offset),
                                              _lib.ptr(y), _lib.ptr(ws), nb, _lib.current_stream(x.device))
        _lib.check(st, "dcn_layer_forward")
        return (y, offset, ws) if keep_workspace else (y, offset)

    def layer_backward(self, x, offset, offset_weight, weight, dy, want_dx=True, want_dow=True, want_dob=False,
                       want_dw=True, want_dbias=False, x_channels_last: Optional[torch.Tensor] = None):
        """Gradients of the layer: (dx, doffset_weight, doffset_bias, dweight, dbias); dx includes the path
        through the offsets."""
        x = self._act(x, "input")
        weight = _prep(weight, "weight", x)
        offset_weight = _prep(offset_weight, "offset_weight", x)
        offset = _prep(offset, "offset", x)
        self._check_offset(offset)
        dy = self._act(dy, "grad_output", x)
        dx = self._new_act(x.shape, x) if want_dx else None
        dow = torch.empty_like(offset_weight) if want_dow else None
        dob = torch.empty(self.offset_channels, dtype=x.dtype, device=x.device) if want_dob else None
        dw = torch.empty(self.weight_shape, dtype=x.dtype, device=x.device) if want_dw else None
        db = torch.empty(self.O, dtype=x.dtype, device=x.device) if want_dbias else None
        ws, nb = self._layer_ws(_lib.PASS_BACKWARD)
        with torch.cuda.device(x.device), _Range("dcn_layer_backward"):
            st = _lib.lib().dcn_layer_backward(ctypes.byref(self.p), _lib.ptr(x), _lib.ptr(offset),
                                               _lib.ptr(offset_weight), _lib.ptr(weight), _lib.ptr(dy),
                                               _lib.ptr(x_channels_last), _lib.ptr(dx), _lib.ptr(dow), _lib.ptr(dob),
                                               _lib.ptr(dw), _lib.ptr(db), _lib.ptr(ws), nb,
                                               _lib.current_stream(x.device))
        _lib.check(st, "dcn_layer_backward")
        return dx, dow, dob, dw, db

    def debug_tc_points(self, offset: torch.Tensor, n: int):
        """Coordinates / validity / corner indices of sample ``n`` decoded from the sampling-point entries that the
        tensor-core backward-data kernel of the 2-D deformable operator consumes (bf16 precision)."""
        offset = _prep(offset, "offset")
        dg, kv, ov = self.C // self.p.cpg, self.offset_channels // (self.C // self.p.cpg) // self.ndim, 1
        for s in self.out_size:
            ov *= s
        coords = torch.empty((dg, kv, ov, self.ndim), dtype=offset.dtype, device=offset.device)
        valid = torch.empty((dg, kv, ov), dtype=torch.int32, device=offset.device)
        lo = torch.empty((dg, kv, ov, self.ndim), dtype=torch.int32, device=offset.device)
        hi = torch.empty_like(lo)
        ws, nb = self._ws(_lib.PASS_BACKWARD)
        with torch.cuda.device(offset.device), _Range("dcn_debug_tc_points"):
            st = _lib.lib().dcn_debug_tc_points(ctypes.byref(self.p), _lib.ptr(offset), n, _lib.ptr(coords),
                                                _lib.ptr(valid), _lib.ptr(lo), _lib.ptr(hi), _lib.ptr(ws), nb,
                                                _lib.current_stream(offset.device))
        _lib.check(st, "dcn_debug_tc_points")
        return coords, valid, lo, hi

    def debug_points(self, offset: torch.Tensor, n: int):
        """Coordinates / validity / corner indices of sample ``n`` as the device routine computes them."""
        offset = _prep(offset, "offset")
        dg, kv, ov = self.C // self.p.cpg, self.offset_channels // (self.C // self.p.cpg) // self.ndim, 1
        for s in self.out_size:
            ov *= s
        coords = torch.empty((dg, kv, ov, self.ndim), dtype=offset.dtype, device=offset.device)
        valid = torch.empty((dg, kv, ov), dtype=torch.int32, device=offset.device)
        lo = torch.empty((dg, kv, ov, self.ndim), dtype=torch.int32, device=offset.device)
        hi = torch.empty_like(lo)
        with torch.cuda.device(offset.device), _Range("dcn_debug_points"):
            st = _lib.lib().dcn_debug_points(ctypes.byref(self.p), _lib.ptr(offset), n, _lib.ptr(coords),
                                             _lib.ptr(valid), _lib.ptr(lo), _lib.ptr(hi),
                                             _lib.current_stream(offset.device))
        _lib.check(st, "dcn_debug_points")
        return coords, valid, lo, hi
