"""The FP64 matrix-vector products (one matrix, several, the blocks of a block
preconditioner) at the edges of their 64-column stages and row shares: a single
row, fewer rows than warps, odd columns and row strides, vectors and matrices
off a 16-byte boundary, against numpy.

Tolerance: a sum of n products in any order is within n u sum |m x| of the exact
one (u = 1.1e-16); numpy's own is within the same."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _close(y, M, x):
    bound = 2.0 * (M.shape[1] + 2) * U * (np.abs(M) @ np.abs(x))
    assert (np.abs(y - M @ x) <= bound).all()


@pytest.mark.parametrize("rows,cols,pad,shift", [(1, 1, 0, 0), (1, 64, 0, 0), (3, 63, 0, 0), (7, 65, 1, 1),
                                                 (17, 128, 2, 0), (300, 127, 3, 1), (2369, 130, 0, 1),
                                                 (4737, 66, 6, 0), (1200, 1201, 1, 0)])
def test_one_matrix(rows, cols, pad, shift):
    from fiber3d_b200 import _lib
    rng = np.random.default_rng(rows + cols)
    M, x = rng.normal(size=(rows, cols)), rng.normal(size=cols)
    ld = cols + pad
    buf = torch.full((shift + rows * ld + 2,), float("nan"), dtype=torch.float64, device="cuda")
    Md = buf[shift:shift + rows * ld].view(rows, ld)
    Md[:, :cols] = torch.tensor(M)
    xb = torch.full((cols + 2,), float("nan"), dtype=torch.float64, device="cuda")
    xd = xb[1:1 + cols]
    xd.copy_(torch.tensor(x))
    y = torch.full((rows + 1,), float("nan"), dtype=torch.float64, device="cuda")
    _lib.call("f3d_gemv", _lib.PRECISION["fp64"], _lib.ptr(Md), ld, _lib.ptr(xd), _lib.ptr(y), rows, cols,
              _lib.stream_handle(y.device))
    got = y.cpu().numpy()
    _close(got[:rows], M, x)
    assert np.isnan(got[rows])


@pytest.mark.parametrize("sizes,vec", [([1], 0), ([6, 64, 130, 2], 1), ([7, 63, 65, 129], 0), ([1206, 318], 1)])
def test_several_matrices(sizes, vec):
    from fiber3d_b200 import _lib
    rng = np.random.default_rng(sum(sizes))
    Ms = [rng.normal(size=(n, n)) for n in sizes]
    x = rng.normal(size=sum(sizes))
    i64 = lambda v: torch.tensor(v, dtype=torch.int64, device="cuda")
    off = np.concatenate([[0], np.cumsum(sizes)])
    moff = np.concatenate([[0], np.cumsum([n * n for n in sizes])])
    M = torch.tensor(np.concatenate([m.reshape(-1) for m in Ms]), device="cuda")
    xd, y = torch.tensor(x, device="cuda"), torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
    m, n, o = i64(moff[:-1]), i64(sizes), i64(off[:-1])
    _lib.call("f3d_gemv_batched", _lib.ptr(M), _lib.ptr(m), _lib.ptr(n), _lib.ptr(o), _lib.ptr(o), len(sizes),
              max(sizes), vec, _lib.ptr(xd), _lib.ptr(y), _lib.stream_handle(y.device))
    got = y.cpu().numpy()
    for b, Mb in enumerate(Ms):
        _close(got[off[b]:off[b + 1]], Mb, x[off[b]:off[b + 1]])


@pytest.mark.parametrize("sizes", [[1, 2, 3, 5], [32, 33, 64, 65, 127, 128], [128] * 600])
def test_blocks(sizes):
    from fiber3d_b200.blocklu import BlockLU
    rng = np.random.default_rng(len(sizes))
    blocks = [rng.normal(size=(n, n)) for n in sizes]
    lu = BlockLU(sizes)
    lu.load(blocks)  # the product is with the blocks as they stand
    x = rng.normal(size=sum(sizes))
    y = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
    lu.apply(torch.tensor(x, device="cuda"), y, "fp64")
    got = y.cpu().numpy()
    for b, Mb in enumerate(blocks):
        o = int(lu.voff_h[b])
        _close(got[o:o + sizes[b]], Mb, x[o:o + sizes[b]])


@pytest.mark.parametrize("rows,cols,pad,shift", [(1, 2, 0, 0), (9, 65, 1, 1), (593, 130, 0, 0), (4740, 64, 2, 0)])
def test_product_on_a_part_of_the_sms(rows, cols, pad, shift):
    from fiber3d_b200 import _lib
    rng = np.random.default_rng(rows)
    M, x = rng.normal(size=(rows, cols)), rng.normal(size=cols)
    ld = cols + pad
    buf = torch.zeros(shift + rows * ld + 2, dtype=torch.float64, device="cuda")
    Md = buf[shift:shift + rows * ld].view(rows, ld)
    Md[:, :cols] = torch.tensor(M)
    xd = torch.tensor(x, device="cuda")
    y = torch.full((rows + 1,), float("nan"), dtype=torch.float64, device="cuda")
    _lib.call("f3d_gemv_beside", _lib.ptr(Md), ld, _lib.ptr(xd), _lib.ptr(y), rows, cols,
              _lib.stream_handle(y.device))
    got = y.cpu().numpy()
    _close(got[:rows], M, x)
    assert np.isnan(got[rows])
