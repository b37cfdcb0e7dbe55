"""One FMM handle through point sets of other sizes, depths and leaf fillings
(leaves of one target, of 128 and of 129, one leaf with nearly all): the same
bits as a fresh handle's, since the same kernels add in the same order."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _targets(rng, kind):
    if kind == "one a leaf":
        g = (np.arange(8) + 0.5) / 8.0
        return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    if kind == "129 a leaf":
        g = (np.arange(4) + 0.5) / 4.0
        c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 1, 3)
        return (c + 0.1 * (rng.random((64, 129, 3)) - 0.5)).reshape(-1, 3)
    if kind == "one leaf":
        return np.concatenate([0.01 + 0.1 * rng.random((2000, 3)), rng.random((40, 3))])
    return rng.random((int(kind), 3))


def test_a_reused_handle_gives_a_fresh_handles_bits():
    from fiber3d_b200.fmm import FMM
    rng = np.random.default_rng(11)
    old = FMM(order=4, max_pts=60)
    old.set_box([0.0, 0.0, 0.0], 1.0)
    for kind, ns in [("300", 500), ("129 a leaf", 3000), ("1", 20), ("one a leaf", 9000), ("one leaf", 400),
                     ("128", 3000), ("20000", 9000)]:
        src, trg, f = rng.random((ns, 3)), _targets(rng, kind), rng.normal(size=(ns, 3))
        new = FMM(order=4, max_pts=60)
        new.set_box([0.0, 0.0, 0.0], 1.0)
        got = []
        for h in (old, new):
            h.set_points(src, src, trg)
            got.append(h.evaluate(sl_density=f, dl_normal=f, dl_density=f[::-1].copy()))
        assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1]), kind
        assert old.tree_info() == new.tree_info()
        new.close()
