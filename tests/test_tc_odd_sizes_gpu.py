"""Tensor-core kernels on outputs whose rows are not 16-byte aligned (the forward kernel turns them in shared memory, its
variant that locates points in its producers stores them from registers): ragged tails of positions and channels, K parts
added up.  All gradients beside the output."""
import numpy as np
import pytest

from tests import cases, helpers
from tests.cases import Case

pytestmark = pytest.mark.gpu

ODD = [
    Case("odd_tail", 2, 3, 32, 40, (13, 17), (3, 3), (1, 1), (1, 1), (1, 1), 1, 16, offset_std=2.0, bias=True),
    Case("odd_split_k", 2, 1, 256, 264, (11, 7), (3, 3), (1, 1), (1, 1), (1, 1), 1, 64, offset_std=2.0, bias=True),
    Case("odd_direct", 3, 1, 64, 40, (3, 7, 5), (3, 3, 3), (1, 1, 1), (1, 1, 1), (1, 1, 1), 4, 8, offset_std=1.5, bias=True),
    Case("odd_plain", 2, 2, 24, 72, (15, 11), (3, 3), (1, 1), (1, 1), (1, 1), 1, 24, deformable=False, bias=True),
]


@pytest.mark.parametrize("case", ODD, ids=[c.name for c in ODD])
def test_odd_output_sizes(case):
    tensors = cases.make_inputs(case)
    ours = helpers.run_ours(case, tensors, "bf16")
    ref = helpers.run_oracle(case, tensors, np.float64)
    mask = helpers.lattice_mask(case, tensors[2].numpy()) if case.deformable else None
    for k in ref:
        a, b = ours[k].astype(np.float64), ref[k]
        if k == "doff":
            a, b = np.where(mask, 0, a), np.where(mask, 0, b)
        assert cases.rel_err(a, b) <= 2e-2, (case.name, k)
