"""The batched LU of blocks of up to 256 rows (16-column panels, one row per
thread, tensor-core updates) and the blocked substitution at the sizes where
their tiles end, against scipy.linalg.lu_factor / lu_solve.

Tolerances: LU with partial pivoting of an N(0, 1) matrix of n <= 256 rows
has a backward error of a few n u (2.8e-14 n at most here) and two
factorisations that take the same pivots differ by that times the leading
blocks' condition numbers (below 1e4 for these seeds), 1e-9 at the worst;
solutions likewise."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.linalg as sla
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-9


def _check(blocks):
    from fiber3d_b200.blocklu import BlockLU
    sizes = [len(A) for A in blocks]
    lu = BlockLU(sizes)
    lu.load(blocks)
    lu.factor()
    lu.check()
    rhs = np.random.default_rng(7).normal(size=sum(sizes))
    x = lu.solve(torch.tensor(rhs, device="cuda")).cpu().numpy()
    for b, A in enumerate(blocks):
        o, n = int(lu.voff_h[b]), sizes[b]
        ref, piv = sla.lu_factor(A)
        assert np.array_equal(lu.piv[o:o + n].cpu().numpy(), piv), n
        assert rel_err(lu.block(b).cpu().numpy(), ref) < TOL, n
        assert rel_err(x[o:o + n], sla.lu_solve((ref, piv), rhs[o:o + n])) < TOL, n


@pytest.mark.parametrize("sizes", [[1, 2, 15, 16, 17, 31, 32, 33, 34], [47, 48, 49, 63, 64, 65, 96, 127, 128, 129],
                                   [255, 256, 240, 241, 64, 3], [256], [257, 16]])
def test_sizes_at_the_edges_of_tiles(sizes):
    rng = np.random.default_rng(sum(sizes))
    _check([rng.normal(size=(n, n)) for n in sizes])


@pytest.mark.parametrize("n", [20, 64, 200, 256])
def test_equal_magnitudes_take_the_first_row(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n))
    A[:, 0] = np.where(rng.random(n) < 0.5, 1.0, -1.0)  # every row ties in the first column
    _check([A])


@pytest.mark.parametrize("scale", [1e-300, 1e300])
def test_pivots_near_the_ends_of_the_range(scale):
    # rows and columns far from 1: the pivots divide instead of taking a reciprocal
    rng = np.random.default_rng(3)
    A = rng.normal(size=(40, 40))
    A[:, 5] *= scale
    _check([A])


def test_singular_block_is_reported_and_others_stand():
    from fiber3d_b200.blocklu import BlockLU
    rng = np.random.default_rng(5)
    A = rng.normal(size=(64, 64))
    A[:, 40] = 0.0
    B = rng.normal(size=(128, 128))
    lu = BlockLU([64, 128])
    lu.load([A, B])
    lu.factor()
    assert lu.info.cpu().tolist() == [41, 0]
    assert rel_err(lu.block(1).cpu().numpy(), sla.lu_factor(B)[0]) < TOL
