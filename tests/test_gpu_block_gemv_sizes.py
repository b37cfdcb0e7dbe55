"""The block preconditioner's FP64 product at the edges of the sizes where its
kernel changes (16, 32 and 96 rows) and of its row groups (16 rows by 1, 2 or 4),
aligned and not, against numpy.

Tolerance: a sum of n products in any order is within n u sum |m x| of the exact
one (u = 1.1e-16); numpy's own is within the same."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("sizes", [[1], [3, 1, 16, 2], [15, 16, 8], [17, 1, 16], [31, 32, 5], [33, 32, 1], [47, 48, 49],
                                   [63, 64, 65, 4], [95, 96, 1], [97, 96, 33], [127, 128, 129], [256, 255, 2],
                                   [301], [500, 7], [4] * 700, [24] * 300, [96] * 200])
def test_product_matches_numpy(sizes):
    from fiber3d_b200.blocklu import BlockLU
    rng = np.random.default_rng(sum(sizes))
    blocks = [rng.normal(size=(n, n)) for n in sizes]
    lu = BlockLU(sizes)
    lu.load(blocks)  # the product is with the blocks as they stand
    x = rng.normal(size=sum(sizes))
    y = torch.full((sum(sizes) + 1,), float("nan"), dtype=torch.float64, device="cuda")
    lu.apply(torch.tensor(x, device="cuda"), y, "fp64")
    got = y.cpu().numpy()
    assert np.isnan(got[-1])
    for b, M in enumerate(blocks):
        o, n = int(lu.voff_h[b]), sizes[b]
        bound = 2.0 * (n + 2) * U * (np.abs(M) @ np.abs(x[o:o + n]))
        assert (np.abs(got[o:o + n] - M @ x[o:o + n]) <= bound).all(), n
