"""A solver whose scratch grows (another solver on its mesh opted the mesh into the edge sums) drops the graphs
that were captured with the old one: they hold its address, and its memory is given back."""
from types import SimpleNamespace

import pytest

from manapy_b200 import _lib
from manapy_b200.solvers import AdvectionDiffusionSolver, _Graphs


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_grown_scratch_drops_graphs(precision, monkeypatch):
    size = [80]
    S = object.__new__(AdvectionDiffusionSolver)
    S._dm = SimpleNamespace(nbcells=10, nbnodes=5, device="cpu", struct=None, cell_scratch_size=lambda: size[0],
                            cell_scratch_size_f32c=lambda: size[0])
    S._tiles = S._tab32 = None
    S._graphs = _Graphs()
    if precision == "fp64":
        def step():
            return S._scratch()[0]
    else:
        monkeypatch.setattr(_lib, "call", lambda *a: None)
        S.var = SimpleNamespace(device_bc=SimpleNamespace(struct=None))
        S._w32 = S._lo32 = [None, None]
        S._sign32 = S._dt_dev = S._ns32 = S._params = None
        import torch
        S._cs32 = torch.empty(size[0])

        def step():
            S._call_f32c(0, None, None)
            return S._cs32
    first = step()
    S._graphs.keep("steps", object())
    assert step() is first and S._graphs.get("steps") is not None     # nothing grew
    size[0] = 200
    assert step().numel() == 200
    assert S._graphs.get("steps") is None
