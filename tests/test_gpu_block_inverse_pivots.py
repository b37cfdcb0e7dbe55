"""The pivot rule of the batched block inverses: a row within 2^-16 of the
column's largest magnitude (33 to 128 rows), whatever the block's scale.

Which row was taken shows in the second pivot of [[1, b], [1 + d, (1 + d) b]],
all entries exact in FP64: after row 0 it is (1 + d) b - (1 + d) b = 0, reported
as a zero pivot at step 2; after row 1 it is b minus the product of a rounded
1 / (1 + d) with (1 + d) b, which no rounding makes zero."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,other", [(33, 1), (64, 40), (96, 95), (128, 1), (128, 100)])
@pytest.mark.parametrize("d", [2.0 ** -12, 2.0 ** -13, 2.0 ** -15, 1.5 * 2.0 ** -16])
def test_a_row_smaller_by_more_than_the_bound_is_not_taken(n, other, d):
    from fiber3d_b200.blocklu import BlockLU
    b = 1.0 + 2.0 ** -30
    A = np.eye(n)
    A[0, 0], A[0, 1], A[1, 1] = 1.0, b, 1.0
    if other == 1:
        A[1, 0], A[1, 1] = 1.0 + d, (1.0 + d) * b
    else:  # the pair in rows 0 and `other`, columns 0 and 1; row 1 takes column `other`
        A[other] = 0.0
        A[other, 0], A[other, 1] = 1.0 + d, (1.0 + d) * b
        A[1] = 0.0
        A[1, other] = 1.0
    lu = BlockLU([n])
    lu.load([A])
    lu.invert(fp32=False)
    assert lu.info.cpu().tolist() == [0]


@pytest.mark.parametrize("n", [33, 100, 128])
@pytest.mark.parametrize("scale", [1e-200, 1e-50, 1e50, 1e200])
def test_scaled_blocks_keep_their_pivots(n, scale):
    # Gauss-Jordan with (threshold) partial pivoting of an N(0, 1) matrix, as at scale 1
    from fiber3d_b200.blocklu import BlockLU
    A = np.random.default_rng(n).normal(size=(n, n))
    A[0, 0] = 0.0  # a pivot search that sees no magnitudes takes this row
    lu = BlockLU([n])
    lu.load([scale * A])
    lu.invert(fp32=False)
    lu.check()
    assert rel_err(scale * lu.block(0).cpu().numpy(), np.linalg.inv(A)) < 1e-9
