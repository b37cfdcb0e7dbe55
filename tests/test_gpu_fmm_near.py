"""The FMM's near field at the edges of its tiles (64 sources, 128 targets an
item, few items split over the neighbour leaves): points in the box's inner
cells at depth 2 are all one another's neighbours, so the result is the direct
sum, to the pair sums' tolerance of 1e-12 of its largest value."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _points(rng, n):
    return 0.25 + 0.5 * rng.random((n, 3))


@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("nsl,ndl,nt", [(1, 0, 1), (0, 1, 2), (63, 65, 127), (64, 64, 128), (65, 63, 129),
                                        (500, 700, 1000), (3000, 0, 300), (0, 2000, 3000)])
def test_near_field_is_the_direct_sum(nsl, ndl, nt, tensor):
    from fiber3d_b200 import fmm as F
    from oracle import kernels_np as KN
    rng = np.random.default_rng(nsl + 7 * ndl + 13 * nt)
    sl, dl, trg = _points(rng, nsl), _points(rng, ndl), _points(rng, nt)
    if nsl:
        trg[0] = sl[0]  # a coincident pair is left out
    f, nrm, dens = rng.normal(size=(nsl, 3)), rng.normal(size=(ndl, 3)), rng.normal(size=(ndl, 3))
    h = F.FMM(order=6, max_pts=5000)
    h.set_box([0.0, 0.0, 0.0], 1.0)
    h.set_points(sl if nsl else None, dl if ndl else None, trg)
    assert h.tree_info()["depth"] == 2 and h.tree_info()["m2l_pairs"] == 0
    kw = {"dl_tensor": 2.0 * nrm[:, :, None] * dens[:, None, :]} if tensor else {"dl_normal": nrm, "dl_density": dens}
    u = h.evaluate(sl_density=f if nsl else None, **(kw if ndl else {})).cpu().numpy()
    ref = np.zeros(3 * nt)
    if nsl:
        r = trg[:, None, :] - sl[None, :, :]
        d = np.sqrt((r * r).sum(-1))
        with np.errstate(divide="ignore"):
            i = np.where(d > 0.0, 1.0 / d, 0.0)
        g = (r * f[None]).sum(-1) * i ** 3
        ref += ((f[None] * i[..., None] + g[..., None] * r).sum(1) / (8.0 * np.pi)).reshape(-1)
    if ndl:
        ref += np.asarray(KN.stresslet_kernel_source_target(dl, trg, nrm, dens, epsilon_distance=0.0)).reshape(-1)
    assert rel_err(u, ref) < 1e-12
