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


CHAIN = [
    (Case("exact_3d_many_points", 3, 44, 32, 64, (2, 12, 16), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 2, 32, offset_std=1.0), "exact"),
    (Case("exact_two_groups", 2, 5, 96, 96, (30, 33), (3, 3), (1, 1), (1, 1), (1, 1), 2, 24, offset_std=2.0, bias=True), "exact"),
    (Case("exact_fp64", 2, 2, 39, 39, (16, 12), (3, 3), (2, 2), (1, 1), (1, 1), 1, 39, dtype="float64", offset_std=2.0), "exact"),
    (Case("exact_narrow", 3, 3, 128, 64, (4, 21, 21), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 1, 16, offset_std=1.0), "exact"),
    (Case("bf16_plane", 2, 4, 64, 64, (40, 44), (3, 3), (1, 1), (1, 1), (1, 1), 1, 32, offset_std=2.0, bias=True), "bf16"),
    (Case("bf16_split", 2, 1, 256, 256, (50, 41), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0), "bf16"),
    (Case("bf16_3d", 3, 6, 32, 48, (4, 14, 14), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 1, 32, offset_std=1.0), "bf16"),
]


def test_calls_in_a_row_wait_for_their_own_prologue():
    """The kernels of a call become resident while the one before them still runs, and must not read what it writes before
    it has finished.  Calls of different problems in a row, over workspaces whose memory holds zeros instead of the last
    call's values (a point read too early then is a wrong one, but an address within the input): the same bits as each call
    alone."""
    import ctypes
    from deform_conv3d_pytorch_op_b200 import _lib
    made = []
    for case, precision in CHAIN:
        tensors = [None if t is None else t.cuda() for t in cases.make_inputs(case)]
        p = _lib.make_problem(case.ndim, tensors[0].dtype, case.N, case.C, case.O, case.in_size, case.kernel, case.stride,
                              case.pad, case.dil, case.G, case.cpg, True, False, True,
                              _lib.PREC_BF16 if precision == "bf16" else _lib.PREC_EXACT)
        sizes = [_lib.lib().dcn_workspace_bytes(ctypes.byref(p), k) for k in (_lib.PASS_FORWARD, _lib.PASS_BACKWARD)]
        made.append((case, precision, tensors, sizes))

    def step(case, precision, tensors, sizes, alone):
        x, w, off, dy, b = tensors
        x, w = x.detach().requires_grad_(True), w.detach().requires_grad_(True)
        for n in sizes[:1]:
            torch.zeros(n, dtype=torch.uint8, device="cuda")          # freed at once: the memory of the next workspace
        y = _forward(case, (x, w, off, dy, b), precision)
        if alone:
            torch.cuda.synchronize()
        torch.zeros(sizes[1], dtype=torch.uint8, device="cuda")
        dw, dx = torch.autograd.grad(y, (w, x), dy)
        if alone:
            torch.cuda.synchronize()
        return y.detach(), dw, dx

    want = [step(*m, True) for m in made]
    for _ in range(15):
        got = [step(*m, False) for m in made]
        for (case, precision, _, _), a, b in zip(made, got, want):
            assert torch.equal(a[0], b[0]), case.name
            assert torch.equal(a[1], b[1]), case.name
            scale = float(b[2].abs().max())
            assert float((a[2] - b[2]).abs().max()) <= (2e-2 if precision == "bf16" else 1e-4) * scale, case.name
