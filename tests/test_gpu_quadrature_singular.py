"""A surface whose local systems are singular: reported, and the elimination
goes on as if a zero pivot were 1, so the weights stay finite.

Around each face's midpoint of a tetrahedron stand 80 copies of one node (of no
triangle), its 80 nearest.  With every projected centre the same point c,
|c| < 1, the system is [0 P; P^T 0] with 80 equal rows p = (1, c_x, c_y, ...) in
P: column 0 has its largest entry, 1, in the constant's row, which takes columns
1 to 79 to exact zeros (1 is its own reciprocal), zero pivots all.  The other
factors are 0 and the back substitution's quotients are by 1."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_singular_systems_are_reported_and_weights_finite():
    from fiber3d_b200 import _lib
    corners = np.array([[1.0, 1.1, 0.9], [-1.0, -0.9, 1.1], [-1.1, 1.0, -1.0], [0.9, -1.0, -1.1]])
    tri = np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]], dtype=np.int32)
    extra = [1.2 * corners[t].mean(0) + 0.05 * (corners[t[1]] - corners[t[0]]) for t in tri]
    nodes = np.concatenate([corners, np.repeat(extra, 80, axis=0)])
    n, dev = len(nodes), torch.device("cuda", 0)
    X, T = torch.tensor(nodes, device=dev), torch.tensor(tri, device=dev)
    G, w = 2.0 * X, torch.zeros(n, dtype=torch.float64, device=dev)
    size = ctypes.c_size_t(0)
    _lib.call("f3d_surface_quadrature_workspace_bytes", n, len(tri), ctypes.byref(size))
    ws = torch.empty(size.value, dtype=torch.uint8, device=dev)
    _lib.call("f3d_surface_quadrature", _lib.ptr(X), n, _lib.ptr(T), len(tri), _lib.ptr(G), _lib.ptr(w), None,
              _lib.ptr(ws), size.value, _lib.stream_handle(dev))
    assert _lib.device_error(dev) == _lib.F3D_ERR_SINGULAR
    got = w.cpu().numpy()
    assert np.isfinite(got).all() and (got[4:] != 0.0).any()
