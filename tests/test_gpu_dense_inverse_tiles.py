"""The dense inverse at the edges of its update's tiles (64 x 128, shared out
to two CTAs per SM): sizes whose last block has one row, sizes just below and
above the one where a CTA takes a second tile (13 blocks of 128 on 148 SMs),
and row strides beyond the padded square, against numpy.linalg.inv.

Tolerance: with M = diag(+-8..12) + N(0, 1) / sqrt(m) the random part's norm is
about 2, so the condition number is below 14 / 6; an entry collects m rounded
updates, u sqrt(m) condition^2 = 1.1e-16 x 43 x 5.4 = 2.6e-14 in the Frobenius
norm for m = 1800, and 1e-13 leaves a factor 4."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,extra", [(64, 2), (65, 0), (255, 66), (257, 0), (1536, 2), (1537, 130), (1793, 0)])
def test_inverse_matches_numpy(m, extra):
    from fiber3d_b200.hydro import dense_inverse, dense_inverse_ld
    rng = np.random.default_rng(m)
    M = np.diag(rng.uniform(8.0, 12.0, m) * rng.choice([-1.0, 1.0], m)) + rng.normal(size=(m, m)) / np.sqrt(m)
    n = dense_inverse_ld(m)
    A = torch.full((n, n + extra), np.nan, dtype=torch.float64, device="cuda")
    A[:m, :m] = torch.as_tensor(M, device="cuda")
    dense_inverse(A, m)
    ref = np.linalg.inv(M)
    assert np.linalg.norm(A[:m, :m].cpu().numpy() - ref) / np.linalg.norm(ref) < 1e-13
    assert torch.equal(A[m:, :n].cpu(), torch.eye(n, dtype=torch.float64)[m:])
    assert torch.isnan(A[:, n:]).all()
