"""A surface whose triangles fill more than one chunk of the quadrature's local
systems (32768): the weights equal the sums of the per-triangle oracle's on a
sample of nodes, and integrate the sphere's constants."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_than_one_chunk_of_triangles():
    from scipy.spatial import ConvexHull
    from fiber3d_b200 import geometry, quadrature
    from oracle import quadrature as OQ
    n, R = 17000, 10.0
    x, _ = geometry.fibonacci_sphere(n, R)
    tri = ConvexHull(x).simplices.astype(np.int32)
    assert len(tri) > 32768
    w, nni = quadrature.surface_quadrature_weights(x, tri, 2.0 * x, device=torch.device("cuda", 0),
                                                   return_neighbors=True)
    w, nni = w.cpu().numpy(), nni.cpu().numpy().astype(np.int64)
    assert abs(w.sum() / (4 * np.pi * R ** 2) - 1) < 1e-9
    # two nodes that have triangles of both chunks among their entries
    t = np.sort(tri.astype(np.int64), axis=1)
    tn = OQ.triangle_normals(x, t)
    en = OQ.edge_normals(t, tn)
    near = {}
    for node in nni[-1][:2]:
        total = 0.0
        for k in np.nonzero((nni == node).any(axis=1))[0]:
            M, rhs, dist = OQ.triangle_system(x, 2.0 * x, t[k], tn[k], en[k], nni[k])
            sol = np.linalg.solve(M, rhs)[:80] * dist
            total += sol[np.nonzero(nni[k] == node)[0][0]]
        near[node] = total
    for node, value in near.items():
        # the noise of these systems at this spacing, as at 12000 nodes (2e-10)
        assert abs(w[node] - value) < 4e-10 * abs(w).max()
