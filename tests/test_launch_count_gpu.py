"""dcn_launch_count and dcn_layer_launch_count state what the device is given: kernels counted by the profiler."""
import ctypes

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from tests import cases
from tests.cases import Case

pytestmark = pytest.mark.gpu

CASES = [
    Case("plane", 2, 2, 32, 40, (13, 16), (3, 3), (1, 1), (1, 1), (1, 1), 1, 16, offset_std=1.5),
    Case("split", 2, 1, 64, 64, (20, 20), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=1.5),
    Case("large_plane", 2, 1, 16, 16, (101, 96), (3, 3), (2, 2), (1, 1), (1, 1), 1, 16, offset_std=1.5),
    Case("three_d", 3, 1, 32, 32, (3, 9, 8), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 2, 16, offset_std=1.0),
    Case("plain", 2, 2, 32, 40, (13, 16), (3, 3), (1, 1), (1, 1), (1, 1), 1, 32, deformable=False),
    Case("plain_split", 2, 1, 64, 128, (20, 20), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, deformable=False),
    Case("plain_stride", 2, 2, 32, 40, (13, 16), (3, 3), (2, 2), (1, 1), (1, 1), 1, 32, deformable=False),
    Case("tiny", 2, 1, 4, 4, (6, 6), (3, 3), (1, 1), (1, 1), (1, 1), 1, 2, offset_std=1.0),
    Case("short", 2, 4, 2, 4, (64, 64), (3, 3), (1, 1), (1, 1), (1, 1), 1, 2, offset_std=1.0),
]


def _launched(fn):
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    return sum(e.count for e in p.key_averages() if "dcn::" in e.key)


@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("precision", ["exact", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=[c.name for c in CASES])
def test_launch_counts(case, precision, channels_last):
    import deform_conv3d_pytorch_op_b200 as dcn
    from deform_conv3d_pytorch_op_b200 import _lib
    if precision == "bf16" and case.name in ("tiny", "short"):
        pytest.skip("channel counts that bf16 refuses")
    if precision == "exact" and channels_last:
        pytest.skip("exact is channel-first")
    x, w, off, dy, _ = [None if t is None else t.cuda() for t in cases.make_inputs(case)]
    if channels_last:
        fmt = torch.channels_last if case.ndim == 2 else torch.channels_last_3d
        x, dy = x.contiguous(memory_format=fmt), dy.contiguous(memory_format=fmt)
    op = dcn.Op(x, w, case.stride, case.pad, case.dil, case.cpg, case.G, deformable=case.deformable,
                std_size_rule=not case.deformable, precision=precision)
    count = lambda which: _lib.lib().dcn_launch_count(ctypes.byref(op.p), which)
    y, ws = op.forward(x, off, w, keep_workspace=True)
    assert _launched(lambda: op.forward(x, off, w)) == count(_lib.PASS_FORWARD)
    assert _launched(lambda: op.backward_data(x, off, w, dy)) == count(_lib.PASS_BACKWARD_DATA)
    assert _launched(lambda: op.backward_weight(x, off, dy)) == count(_lib.PASS_BACKWARD_WEIGHT)
    assert _launched(lambda: op.backward(x, off, w, dy)) == count(_lib.PASS_BACKWARD)
    assert _launched(lambda: op.backward(x, off, w, dy, x_channels_last=ws)) == count(_lib.PASS_BACKWARD)
    if case.deformable and case.dil == (1,) * case.ndim:
        layer = lambda which: _lib.lib().dcn_layer_launch_count(ctypes.byref(op.p), which)
        ow = torch.randn(op.offset_weight_shape(), device="cuda") * 0.01
        y, offsets = op.layer_forward(x, ow, None, w)
        assert _launched(lambda: op.layer_forward(x, ow, None, w)) == layer(_lib.PASS_FORWARD)
        assert _launched(lambda: op.layer_backward(x, offsets, ow, w, dy)) == layer(_lib.PASS_BACKWARD)
