"""Several FP64 products in one launch on both sides of the rule that takes four
rows at a time (2.1 rows a warp over three CTAs of eight warps per SM), with
sizes that leave one, two or three rows in the last group, against numpy.

Tolerance: a sum of n products in any order is within n u sum |m x| of the exact
one (u = 1.1e-16); numpy's own is within the same."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("sizes,vec", [([130] * 57, 1), ([130] * 58, 1), ([129] * 58, 0), ([131, 1, 2, 3] * 30, 0),
                                       ([306] * 24, 1), ([306, 2, 64] * 13, 1), ([1206] * 7, 1), ([1205] * 7, 0),
                                       ([5] * 1700, 0), ([2] * 6000, 1)])
def test_products_match_numpy(sizes, vec):
    from fiber3d_b200 import _lib
    rng = np.random.default_rng(len(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)])
    moff = np.concatenate([[0], np.cumsum([n * n for n in sizes])])
    Mh, xh = rng.normal(size=moff[-1]), rng.normal(size=off[-1])
    i64 = lambda v: torch.tensor(v, dtype=torch.int64, device="cuda")
    M, x = torch.tensor(Mh, device="cuda"), torch.tensor(xh, device="cuda")
    y = torch.full((int(off[-1]) + 1,), float("nan"), dtype=torch.float64, device="cuda")
    m, n, o = i64(moff[:-1]), i64(sizes), i64(off[:-1])
    _lib.call("f3d_gemv_batched", _lib.ptr(M), _lib.ptr(m), _lib.ptr(n), _lib.ptr(o), _lib.ptr(o), len(sizes),
              max(sizes), vec, _lib.ptr(x), _lib.ptr(y), _lib.stream_handle(y.device))
    got = y.cpu().numpy()
    assert np.isnan(got[-1])
    for b, k in enumerate(sizes):
        A, xb = Mh[moff[b]:moff[b + 1]].reshape(k, k), xh[off[b]:off[b + 1]]
        bound = 2.0 * (k + 2) * U * (np.abs(A) @ np.abs(xb))
        assert (np.abs(got[off[b]:off[b + 1]] - A @ xb) <= bound).all(), (b, k)
