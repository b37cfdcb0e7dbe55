"""Batched block inverses at the edges of the blocked kernels (64, 96 and 128
rows, 16-column panels, 4-column sub-panels), odd sizes among them, against
numpy.linalg.inv.

Tolerance: Gauss-Jordan with (threshold) partial pivoting of an N(0, 1) matrix
of n <= 128 rows has an error of a few n u (2.8e-14) times the condition
number, below 1e4 for these seeds: 1e-9 at the worst."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.mark.parametrize("sizes", [[33, 34, 47, 48, 49, 63, 64, 1, 16], [65, 80, 81, 95, 96, 64, 7],
                                   [97, 111, 112, 113, 127, 128, 20], [128], [96], [64] * 200, [128] * 150])
def test_inverse_matches_numpy(sizes):
    from fiber3d_b200.blocklu import BlockLU
    rng = np.random.default_rng(sum(sizes) + len(sizes))
    blocks = [rng.normal(size=(n, n)) for n in sizes]
    lu = BlockLU(sizes)
    lu.load(blocks)
    lu.invert(fp32=True)
    lu.check()
    a32 = lu.A32.cpu().numpy()
    for b, A in enumerate(blocks):
        n, o = sizes[b], int(lu.moff_h[b])
        ref = np.linalg.inv(A)
        got = lu.block(b).cpu().numpy()
        assert rel_err(got, ref) < TOL, n
        assert np.array_equal(a32[o:o + n * n].reshape(n, n), got.astype(np.float32))


@pytest.mark.parametrize("n,k", [(40, 1), (96, 50), (100, 100), (128, 17)])
def test_zero_pivot_is_reported_at_its_step(n, k):
    from fiber3d_b200.blocklu import BlockLU
    A = np.eye(n)
    A[k - 1, k - 1] = 0.0
    lu = BlockLU([n, n])
    lu.load([A, np.eye(n)])
    lu.invert(fp32=False)
    assert lu.info.cpu().tolist() == [k, 0]
