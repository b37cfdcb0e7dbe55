"""The substitution of many small systems on both sides of the rule that hands
them to one warp each (batches of more than 1000 systems up to 12 rows, 1500
below 32, 2500 below 64, 4000 of 32 and below 96, 5000 up to 160, all per wave),
odd and mixed sizes, against numpy.

Tolerance: with A = N(0, 1) + 3 sqrt(n) I the random part's norm is about
2 sqrt(n), so condition(A) <= 5 / 1; the backward error of LU with partial
pivoting of n <= 160 rows is a few n u (1.8e-14 n u-sums at most), times the
condition number below 1e-12 of the largest unknown."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cycle,count", [([1], 1501), ([7], 1000), ([7], 1001), ([13, 1], 1500), ([13, 1], 1501), (list(range(1, 32)), 3001),
                                         ([32], 4001), ([32, 5], 4000), ([33, 34, 40, 63, 2], 2501),
                                         ([48], 2500), ([64, 9], 5001), ([65, 3], 4001), ([96, 65, 3], 5003), ([20], 20000),
                                         ([160, 8, 12, 4], 5001), ([161, 8], 5001)])
def test_many_small_systems(cycle, count):
    from fiber3d_b200.blocklu import BlockLU
    rng = np.random.default_rng(count + len(cycle))
    sizes = [cycle[k % len(cycle)] for k in range(count)]
    lu = BlockLU(sizes)
    A = {}
    host = np.empty(lu.A.numel())
    for b, n in enumerate(sizes):
        o = int(lu.moff_h[b])
        host[o:o + n * n] = (rng.normal(size=(n, n)) + 3.0 * np.sqrt(n) * np.eye(n)).ravel()
        if b % 97 == 0 or b >= count - 3:
            A[b] = host[o:o + n * n].reshape(n, n).copy()
    lu.A[:len(host)].copy_(torch.tensor(host))
    lu.factor()
    lu.check()
    rhs = rng.normal(size=lu.nvec)
    for _ in range(2):  # the queue's counters return to zero
        x = lu.solve(torch.tensor(rhs, device="cuda")).cpu().numpy()
        assert np.isfinite(x).all()
        for b, M in A.items():
            o = int(lu.voff_h[b])
            assert rel_err(x[o:o + len(M)], np.linalg.solve(M, rhs[o:o + len(M)])) < 1e-12, (b, len(M))
