"""The channels-last kernels of the exact precision at the edges of their tiles and segments, against the float64
oracle: vectors padded within a segment, single-channel vectors, deformable groups over several convolution groups,
every tile height, two output-channel tiles, ragged positions, parts of the K range, fp64."""
import ctypes

import numpy as np
import pytest

from tests import cases, helpers
from tests.cases import Case

pytestmark = pytest.mark.gpu

EDGES = [
    Case("pad5", 2, 2, 40, 33, (21, 19), (3, 3), (1, 1), (1, 1), (1, 1), 1, 5, offset_std=2.0, bias=True),
    Case("pad3_two_tiles", 3, 2, 12, 130, (3, 9, 11), (3, 3, 3), (1, 2, 1), (1, 1, 1), (1, 1, 1), 1, 3, offset_std=1.5),
    Case("dg_over_groups", 2, 3, 64, 64, (17, 15), (3, 3), (1, 1), (2, 2), (2, 2), 4, 32, offset_std=3.0, bias=True),
    Case("single_channels", 2, 13, 32, 20, (23, 21), (3, 3), (2, 1), (1, 1), (1, 1), 1, 2, offset_std=1.0),
    Case("tall_tile_split_k", 2, 1, 96, 128, (13, 10), (3, 3), (1, 1), (1, 1), (1, 1), 1, 48, offset_std=2.0, bias=True),
    Case("three_d_groups", 3, 3, 32, 192, (4, 9, 9), (3, 3, 3), (1, 2, 2), (2, 2, 2), (2, 2, 2), 2, 16, offset_std=2.0),
    Case("plain_stride", 2, 5, 20, 36, (33, 27), (3, 3), (2, 2), (1, 1), (1, 1), 2, 20, deformable=False, bias=True),
    Case("plain_dilated", 2, 2, 18, 97, (25, 18), (3, 3), (1, 1), (2, 2), (2, 2), 1, 18, deformable=False),
    Case("fp64_pad", 2, 2, 12, 70, (9, 8), (3, 3), (1, 1), (1, 1), (1, 1), 2, 3, dtype="float64", offset_std=2.0, bias=True),
    Case("fp64_single", 3, 1, 4, 6, (3, 5, 4), (2, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 1, 1, dtype="float64", offset_std=1.5),
]


@pytest.mark.parametrize("case", EDGES, ids=[c.name for c in EDGES])
def test_exact_kernels_at_tile_and_segment_edges(case):
    from deform_conv3d_pytorch_op_b200 import _lib
    tensors = cases.make_inputs(case)
    p = _lib.make_problem(case.ndim, tensors[0].dtype, case.N, case.C, case.O, case.in_size, case.kernel, case.stride,
                          case.pad, case.dil, case.G, case.cpg, case.deformable, not case.deformable)
    assert _lib.lib().dcn_workspace_bytes(ctypes.byref(p), _lib.PASS_BACKWARD) > 0         # these kernels are the ones taken
    ours = helpers.run_ours(case, tensors, "exact")
    ref = helpers.run_oracle(case, tensors, np.float64)
    mask = helpers.lattice_mask(case, tensors[2].numpy()) if case.deformable else None
    tol = 1e-4 if case.dtype == "float32" else 1e-10
    for k in ref:
        a, b = ours[k].astype(np.float64), ref[k]
        if k == "doff":
            a, b = np.where(mask, 0, a), np.where(mask, 0, b)
        assert cases.rel_err(a, b) <= tol, (case.name, k)


@pytest.mark.parametrize("kind", ["deform", "plain", "layer"])
def test_a_call_without_room_for_its_workspace(kind):
    """The exact precision needs no workspace: where the allocator has no room for one, a call runs on the kernels that do
    without.  The room is limited through torch's allocator, to what the outputs take."""
    import torch
    import deform_conv3d_pytorch_op_b200 as dcn
    g = torch.Generator(device="cuda").manual_seed(1)
    n, c, s = 16, 96, 64                                              # every tensor of note over the 20 MB of a shared segment

    def leaf(*shape, std=1.0):
        return (torch.randn(shape, generator=g, device="cuda") * std).requires_grad_(True)

    x, w = leaf(n, c, s, s), leaf(c, c, 3, 3, std=0.05)
    dy = torch.randn((n, c, s, s), generator=g, device="cuda")
    if kind == "deform":
        args = [x, leaf(n, 72, s, s), w]
        fn = lambda: dcn.ConvOffset2dFunction.apply(*args, None, 1, 1, 1, 24, 1)
    elif kind == "plain":
        args = [x, w]
        fn = lambda: dcn.Conv2dFunction.apply(*args, None, 1, 1, 1)
    else:
        # offsets of 0.5 with a deviation of 0.06: rounding carries no point over the integer lattice, where values jump
        args = [x, leaf(72, c, 3, 3, std=0.002), w]
        half = torch.full((72,), 0.5, device="cuda")
        fn = lambda: dcn.DeformLayerFunction.apply(x, args[1], half, w, None, 1, 1, 1, 24, 1)
    y = fn()
    want = (y.detach(),) + torch.autograd.grad(y, args, dy)
    del y
    mb = lambda *ts: sum((t.numel() * 4 + 2097151) // 2097152 * 2097152 for t in ts)
    offsets = n * 72 * s * s * 4 if kind == "layer" else 0
    total = torch.cuda.get_device_properties(0).total_memory

    def limit(room):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / total)

    try:
        limit(mb(x) + offsets + (4 << 20))
        y = fn()
        # the gradients, the offset gradient of a layer, and a segment of 20 MB for the small ones
        limit(mb(*args) + offsets + (24 << 20))
        got = (y.detach(),) + torch.autograd.grad(y, args, dy)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert cases.rel_err(a.cpu().numpy(), b.cpu().numpy()) <= 1e-4
