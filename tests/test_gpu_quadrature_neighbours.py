"""The quadrature's nearest neighbours against numpy, exactly: surfaces of the
smallest size, an odd number of triangles pairs' worth, equal distances beyond
what one collection pass holds, and node orders that put a triangle's
neighbours into few of the kernel's groups."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(nodes, tri, k=80):
    t = np.sort(tri, axis=1)
    mid = ((nodes[t[:, 0]] + nodes[t[:, 1]]) + nodes[t[:, 2]]) / 3.0
    d = mid[:, None, :] - nodes[None, :, :]
    d2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
    idx = np.broadcast_to(np.arange(len(nodes)), d2.shape)
    return np.lexsort((idx, d2), axis=1)[:, :k]


def _sphere(n, order):
    from scipy.spatial import ConvexHull
    from fiber3d_b200 import geometry
    x, _ = geometry.fibonacci_sphere(n, 10.0)
    if order == "near first":  # nodes of one cap fill whole runs of indices
        x = x[np.argsort(np.linalg.norm(x - x[n // 3], axis=1))]
    elif order == "strided":  # neighbours 256 indices apart: all in one thread's group
        p = np.argsort(np.linalg.norm(x - x[n // 3], axis=1))
        out = np.empty_like(x)
        out[np.argsort(np.arange(n) % 256, kind="stable")] = x[p]
        x = out
    return x, ConvexHull(x).simplices.astype(np.int32)


@pytest.mark.parametrize("n,order", [(80, "lattice"), (82, "lattice"), (300, "lattice"), (2000, "lattice"),
                                     (2000, "near first"), (2000, "strided"), (6000, "strided")])
def test_neighbours_exact(n, order):
    from fiber3d_b200.quadrature import surface_quadrature_weights
    x, tri = _sphere(n, order)
    _, nni = surface_quadrature_weights(x, tri, 2.0 * x, device=torch.device("cuda", 0), return_neighbors=True)
    assert np.array_equal(nni.cpu().numpy(), _reference(x, tri))
