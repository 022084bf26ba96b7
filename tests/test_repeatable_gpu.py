"""Forward passes give the same bits on every call, also where the K range of a tile is computed in parts by several
CTAs: the parts are added in a fixed order, whichever finishes first."""
import numpy as np
import pytest
import torch

from tests import cases, helpers
from tests.cases import Case

pytestmark = pytest.mark.gpu

EXACT = [
    Case("narrow_18_parts", 2, 1, 96, 128, (13, 10), (3, 3), (1, 1), (1, 1), (1, 1), 1, 48, offset_std=2.0, bias=True),
    Case("wide_4_parts", 2, 6, 96, 96, (33, 45), (3, 3), (1, 1), (1, 1), (1, 1), 1, 48, offset_std=2.0, bias=True),
    Case("wide_two_tiles", 2, 2, 64, 200, (49, 50), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0),
    Case("three_d", 3, 2, 32, 72, (4, 9, 7), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 2, 16, offset_std=1.5, bias=True),
    Case("single_channels", 2, 3, 64, 40, (15, 16), (3, 3), (1, 1), (1, 1), (1, 1), 1, 2, offset_std=1.0),
    Case("plain", 2, 2, 48, 72, (20, 19), (3, 3), (1, 1), (1, 1), (1, 1), 1, 48, deformable=False, bias=True),
    Case("fp64", 2, 2, 32, 32, (28, 28), (3, 3), (1, 1), (1, 1), (1, 1), 1, 32, dtype="float64", offset_std=2.0, bias=True),
    Case("fp64_tails", 2, 1, 33, 70, (11, 13), (3, 3), (1, 1), (1, 1), (1, 1), 1, 11, dtype="float64", offset_std=2.0),
]


def _forward(case, tensors, precision):
    import deform_conv3d_pytorch_op_b200 as dcn
    x, w, off, _, b = [None if t is None else t.cuda() for t in tensors]
    if case.deformable:
        fn = dcn.ConvOffset3dFunction if case.ndim == 3 else dcn.ConvOffset2dFunction
        return fn.apply(x, off, w, b, case.stride, case.pad, case.dil, case.cpg, case.G, precision)
    return dcn.Conv2dFunction.apply(x, w, b, case.stride, case.pad, case.dil, case.G, precision)


def _oracle(case, tensors):
    x, w, off, _, b = [None if t is None else t.numpy().astype(np.float64) for t in tensors]
    p = case.problem()
    p.N = case.N
    return helpers.orc.forward(p, x, off, w, b)


@pytest.mark.parametrize("case", EXACT, ids=[c.name for c in EXACT])
def test_exact_forward_is_repeatable(case):
    tensors = cases.make_inputs(case)
    first = _forward(case, tensors, "exact")
    tol = 1e-4 if case.dtype == "float32" else 1e-10
    assert cases.rel_err(first.cpu().numpy().astype(np.float64), _oracle(case, tensors)) <= tol
    assert all(torch.equal(_forward(case, tensors, "exact"), first) for _ in range(20))


BF16 = [
    Case("three_chunks_a_part", 2, 1, 64, 64, (19, 21), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0, bias=True),
    Case("two_halves", 2, 2, 128, 136, (40, 40), (3, 3), (1, 1), (1, 1), (1, 1), 1, 32, offset_std=2.0, bias=True),
    Case("tail_two_groups", 2, 4, 128, 96, (49, 50), (3, 3), (1, 1), (1, 1), (1, 1), 2, 64, offset_std=2.0, bias=True),
    Case("tail_three_blocks", 2, 4, 64, 648, (50, 48), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0, bias=True),
    Case("three_d", 3, 3, 64, 40, (2, 7, 7), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 1, 64, offset_std=1.0),
    Case("plain", 2, 2, 64, 192, (23, 21), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, deformable=False, bias=True),
]


@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("case", BF16, ids=[c.name for c in BF16])
def test_bf16_forward_is_repeatable(case, channels_last):
    tensors = list(cases.make_inputs(case))
    ref = _oracle(case, tensors)
    if channels_last:
        tensors[0] = tensors[0].contiguous(memory_format=torch.channels_last if case.ndim == 2 else torch.channels_last_3d)
    first = _forward(case, tensors, "bf16")
    assert cases.rel_err(first.cpu().numpy().astype(np.float64), ref) <= 2e-2
    assert all(torch.equal(_forward(case, tensors, "bf16"), first) for _ in range(20))


def test_bf16_plain_input_gradient_is_repeatable():
    """The input gradient of a stride-1 plain convolution is a forward pass of the transposed one, split like it."""
    import deform_conv3d_pytorch_op_b200 as dcn
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((2, 64, 23, 21), generator=g, device="cuda").requires_grad_(True)
    w = torch.randn((192, 64, 3, 3), generator=g, device="cuda") * 0.05
    dy = torch.randn((2, 192, 23, 21), generator=g, device="cuda")

    def dx():
        return torch.autograd.grad(dcn.Conv2dFunction.apply(x, w, None, 1, 1, 1, 1, "bf16"), x, dy)[0]

    first = dx()
    want = torch.nn.grad.conv2d_input(x.shape, w.double(), dy.double(), padding=1)
    assert cases.rel_err(first.cpu().numpy().astype(np.float64), want.cpu().numpy()) <= 2e-2
    assert all(torch.equal(dx(), first) for _ in range(20))
