"""The order of the two streams in pc_matvec, made decisive: other vectors at each
call, results set to NaN before it, a delay of about a millisecond ahead of the
periphery's product on its stream (a matvec that does not wait for it reads NaN)
and one ahead of writing x on the calling stream (a product that does not wait
reads NaN); eager, on another stream, and replayed from a graph.

Tolerance: as for one call against the two operators one after the other (the
product with the inverse adds m <= 1200 terms in another order): 1e-12 of z,
1e-11 of A z."""
from __future__ import annotations

import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu

DELAY = 2_000_000  # clock cycles


@pytest.fixture(scope="module")
def system():
    from fiber3d_b200.geometry import hydro_step_problem
    from fiber3d_b200.hydro import HydroSystem
    return HydroSystem(hydro_step_problem(seed=6, nfib=40, nbody=1, body_nodes=80, nshell=400))


@pytest.fixture
def delayed(system, monkeypatch):
    from fiber3d_b200 import hydro
    plain = hydro.ShellOperator.apply

    def apply(self, x, y, storage="fp64", beside=False):
        if beside:
            torch.cuda._sleep(DELAY)
        return plain(self, x, y, storage, beside)

    monkeypatch.setattr(hydro.ShellOperator, "apply", apply)
    monkeypatch.setattr(system, "product_beside_sum", lambda: True)
    return system


def _vectors(system, k):
    gen = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn(system.size, dtype=torch.float64, device="cuda", generator=gen)
    z, w = torch.empty_like(x), torch.empty_like(x)
    system.pc(x, z)
    system.matvec(z, w)
    torch.cuda.synchronize()
    return x, z, w


@pytest.mark.parametrize("how", ["eager", "other stream", "graph"])
def test_every_call_waits_both_ways(delayed, how):
    cases = [_vectors(delayed, k) for k in range(4)]
    x, z, w = (torch.empty_like(cases[0][0]) for _ in range(3))
    graph = None
    if how == "graph":
        x.copy_(cases[0][0])
        warm = torch.cuda.Stream()
        warm.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(warm):
            delayed.pc_matvec(x, z, w)
        torch.cuda.current_stream().wait_stream(warm)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            delayed.pc_matvec(x, z, w)
    s = torch.cuda.Stream() if how == "other stream" else torch.cuda.current_stream()
    s.wait_stream(torch.cuda.current_stream())
    for x1, z1, w1 in cases:
        with torch.cuda.stream(s):
            for t in (x, z, w):
                t.fill_(float("nan"))
            torch.cuda._sleep(DELAY)
            x.copy_(x1)
            if graph is not None:
                graph.replay()
            else:
                delayed.pc_matvec(x, z, w)
            got = z.clone(), w.clone()
        s.synchronize()
        assert rel_err(got[0].cpu().numpy(), z1.cpu().numpy()) < 1e-12
        assert rel_err(got[1].cpu().numpy(), w1.cpu().numpy()) < 1e-11


def test_vectors_are_the_callers_again_after_a_raise(delayed, monkeypatch):
    from fiber3d_b200 import hydro
    x, z0, w = _vectors(delayed, 9)
    z = torch.zeros_like(x)

    def fail(self, *a):
        raise RuntimeError("no fibers today")

    monkeypatch.setattr(hydro.HydroSystem, "_pc_bodies_fibers", fail)
    with pytest.raises(RuntimeError, match="no fibers"):
        delayed.pc_matvec(x, z, w)
    z.fill_(7.0)  # after the delayed product, not before it
    torch.cuda.synchronize()
    assert (z == 7.0).all()
