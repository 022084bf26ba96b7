"""Splits of the tensor-core forward tiles along K: every tile in pieces of three chunks, and the tail of an uneven grid
where it lies in the last (group, channel block), with channel-first and channels-last outputs.  And the 2-D backward-data
kernel with fewer taps than epilogue warps per quarter."""
import numpy as np
import pytest
import torch

from tests import cases, helpers
from tests.cases import Case

pytestmark = pytest.mark.gpu

SPLITS = [
    Case("three_chunks", 2, 1, 64, 64, (19, 21), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0, bias=True),
    # 2 groups x 77 position tiles: the six tiles of the second wave lie in the last group
    Case("tail_two_groups", 2, 4, 128, 96, (49, 50), (3, 3), (1, 1), (1, 1), (1, 1), 2, 64, offset_std=2.0, bias=True),
    # 2 channel blocks x 75 position tiles
    Case("tail_two_blocks", 2, 4, 64, 320, (50, 48), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0, bias=True),
]


@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("case", SPLITS, ids=[c.name for c in SPLITS])
def test_forward_splits(case, channels_last):
    import deform_conv3d_pytorch_op_b200 as dcn
    tensors = cases.make_inputs(case)
    x, w, off, _, b = (t.cuda() for t in tensors)
    if channels_last:
        x = x.contiguous(memory_format=torch.channels_last)
    y = dcn.ConvOffset2dFunction.apply(x, off, w, b, case.stride, case.pad, case.dil, case.cpg, case.G, "bf16")
    xn, wn, on, dyn, bn = (t.numpy().astype(np.float64) for t in tensors)
    p = case.problem()
    p.N = case.N
    ref = helpers.orc.forward(p, xn, on, wn, bn)
    assert cases.rel_err(y.cpu().numpy().astype(np.float64), ref) <= 2e-2


FEW_TAPS = [
    Case("one_tap", 2, 2, 48, 40, (21, 20), (1, 1), (1, 1), (0, 0), (1, 1), 1, 24, offset_std=1.5, bias=True),
    Case("two_taps", 2, 1, 32, 72, (30, 23), (1, 2), (1, 1), (0, 0), (1, 1), 2, 16, offset_std=1.5),
    Case("three_taps", 2, 1, 16, 16, (25, 24), (3, 1), (1, 1), (1, 0), (1, 1), 1, 16, offset_std=1.5),
]


@pytest.mark.parametrize("case", FEW_TAPS, ids=[c.name for c in FEW_TAPS])
def test_backward_data_with_few_taps(case):
    import deform_conv3d_pytorch_op_b200 as dcn
    tensors = cases.make_inputs(case)
    ours = helpers.run_ours(case, tensors, "bf16")
    dcn.check_status()                       # no bounded wait gave up
    ref = helpers.run_oracle(case, tensors, np.float64)
    mask = helpers.lattice_mask(case, tensors[2].numpy())
    for k in ref:
        a, b = ours[k].astype(np.float64), ref[k]
        if k == "doff":
            a, b = np.where(mask, 0, a), np.where(mask, 0, b)
        assert cases.rel_err(a, b) <= 2e-2, (case.name, k)
