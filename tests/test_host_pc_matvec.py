"""HydroSystem.pc_matvec honours operators that a subclass or an instance puts in
the place of its own, and solve_system asks the system itself for pc_matvec, not
an object that the system passes attributes on from.  No device: the operators
are recorded."""
from __future__ import annotations

import types

import pytest
import torch


def _system(cls, calls):
    from fiber3d_b200 import hydro
    s = cls.__new__(cls)
    s.product_beside_sum = lambda: True
    s.device, s._side = torch.device("cpu"), None
    s.shell = hydro.ShellOperator.__new__(hydro.ShellOperator)
    return s


def test_a_subclass_with_its_own_operators():
    from fiber3d_b200.hydro import HydroSystem
    calls = []

    class Own(HydroSystem):
        def pc(self, x, y, precision="fp64"):  # returns nothing
            calls.append(("pc", x, y))

        def matvec(self, x, y, precision="fp64"):  # knows no `join`
            calls.append(("matvec", x, y))
            return y

    assert _system(Own, calls).pc_matvec("x", "z", "w") == "w"
    assert calls == [("pc", "x", "z"), ("matvec", "z", "w")]


@pytest.mark.parametrize("where", ["pc", "matvec", "shell"])
def test_an_instance_with_its_own_operators(where, monkeypatch):
    from fiber3d_b200 import hydro
    calls = []
    s = _system(hydro.HydroSystem, calls)
    if where == "shell":
        s.nS, s.inner_shell_pc = 1, "fp32"
        s.shell.apply = lambda x, y, storage="fp64": calls.append(("shell", x, y))
        monkeypatch.setattr(hydro.HydroSystem, "_pc_bodies_fibers", lambda self, x, y, p: calls.append(("rest", x, y)))
        # the class's own matvec, recorded: still its own
        monkeypatch.setattr(hydro.HydroSystem, "matvec", lambda self, x, y, p="fp64": calls.append(("matvec", x, y)))
        s.pc_matvec("x", "z", "w")
        assert calls == [("shell", "x", "z"), ("rest", "x", "z"), ("matvec", "z", "w")]
        return
    other = {"pc": "matvec", "matvec": "pc"}[where]
    setattr(s, where, lambda x, y, precision="fp64": calls.append((where, x, y)))
    monkeypatch.setattr(hydro.HydroSystem, other, lambda self, x, y, p="fp64": calls.append((other, x, y)))
    s.pc_matvec("x", "z", "w")
    assert calls == [("pc", "x", "z"), ("matvec", "z", "w")]


def test_a_system_around_another_keeps_its_operators(monkeypatch):
    from fiber3d_b200 import gmres
    seen = {}

    class Recorder:
        def __init__(self, n, m, dev):
            self.n, self.m = n, m

        def solve(self, matvec, pc, b, **kw):
            seen.update(kw, matvec=matvec, pc=pc)
            return b, 0, 0, []

    class Around:  # passes on what it does not have
        def __init__(self, inner):
            self.inner = inner

        def __getattr__(self, name):
            return getattr(self.inner, name)

        def pc(self, x, y, precision="fp64"):
            return "own"

    inner = types.SimpleNamespace(device="cpu", size=1, rhs="b", pc_matvec=lambda *a: "inner", matvec=None, pc=None,
                                  _gmres=None)
    monkeypatch.setattr(gmres, "DeviceGMRES", Recorder)
    gmres.solve_system(Around(inner))
    assert seen["pc_matvec"] is None and seen["pc"]("x", "y") == "own"
