"""The preconditioner and the matvec of an Arnoldi step in one call, with the
periphery's product on a stream of its own beside the Oseen sum, against one
after the other: called directly, on another stream, and in a solve (captured in
a graph and not).

Tolerance: the two products with the inverse add the same m <= 1200 products in
another order, so z differs by at most 2 m u |M| |x| an entry (u = 1.1e-16): below
1e-12 of |z| for these second-kind inverses, and A z, a sum of terms of z's size,
likewise with a factor 10 for cancellation.  Two solves to a residual of 1e-10
agree to that times the preconditioned system's condition number, below 100."""
from __future__ import annotations

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    from fiber3d_b200.geometry import hydro_step_problem
    from fiber3d_b200.hydro import HydroSystem
    return HydroSystem(hydro_step_problem(seed=5, nfib=40, nbody=1, body_nodes=80, nshell=400))


@pytest.mark.parametrize("other_stream", [False, True])
def test_same_as_one_after_the_other(system, monkeypatch, other_stream):
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(system.size, dtype=torch.float64, device="cuda", generator=gen)
    z0, w0, z, w = (torch.empty_like(x) for _ in range(4))
    system.pc(x, z0)
    system.matvec(z0, w0)
    monkeypatch.setattr(system, "product_beside_sum", lambda: True)
    s = torch.cuda.Stream() if other_stream else torch.cuda.current_stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(5):
            system.pc_matvec(x, z, w)
    torch.cuda.current_stream().wait_stream(s)
    assert rel_err(z.cpu().numpy(), z0.cpu().numpy()) < 1e-12
    assert rel_err(w.cpu().numpy(), w0.cpu().numpy()) < 1e-11


@pytest.mark.parametrize("use_graph", [False, True])
def test_solve(system, monkeypatch, use_graph):
    ref = system.solve(tol=1e-10, use_graph=use_graph)["x"].clone()
    system._gmres = None  # a captured step keeps its route
    monkeypatch.setattr(system, "product_beside_sum", lambda: True)
    res = system.solve(tol=1e-10, use_graph=use_graph)
    system._gmres = None
    assert res["info"] == 0
    assert rel_err(res["x"].cpu().numpy(), ref.cpu().numpy()) < 1e-8


def test_fp32c_takes_the_plain_route(system, monkeypatch):
    monkeypatch.setattr(system, "product_beside_sum", lambda: True)
    monkeypatch.setattr(system.shell, "apply", _no_beside(system.shell.apply))
    x = torch.ones(system.size, dtype=torch.float64, device="cuda")
    system.pc_matvec(x, torch.empty_like(x), torch.empty_like(x), "fp32c")


def _no_beside(apply):
    def f(x, y, storage="fp64", beside=False):
        assert not beside
        return apply(x, y, storage)
    return f
