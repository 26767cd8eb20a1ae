"""Where the device has no memory left for the tables of a step, the solver takes the step that needs none:
the results of a solver that has them, to 1e-12 of the largest value after 6 steps (some hundred rounded
operations a step; equal bits for the steps that share their arithmetic)."""
import numpy as np
import pytest
import torch

from conftest import rel_max
import manapy_b200 as M
from manapy_b200 import meshgen
from manapy_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu


def _domain(dim):
    return M.Domain(dim=dim, mesh=meshgen.square_triangles(14, seed=2) if dim == 2 else meshgen.cube_tetrahedra(5, seed=2))


def _advdiff(dom, dim, precision):
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    for var, a in zip((u, v, z), (0.7, 0.4, 0.3 * (dim - 2))):
        var.face = np.full(len(var.face), a)
        var.interpolate_facetocell()
    w.cell = 1 + 0.2 * np.sin(5 * dom.cells.center[:, 0])
    return [w], M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=2e-3, Dzz=1e-3 * (dim - 2),
                                                                           order=2, cfl=0.4, precision=precision))


def _five(dom, kind):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    x = dom.cells.center
    if kind == "sw":
        vs[0].cell = np.where(x[:, 0] < 0.5, 2.0, 1.0)
        return vs[:4], M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))
    for v, a in zip(vs, (1.0, 1.0, 0.1, 0.1, 2.5)):
        v.cell = a * (1 + 0.1 * np.sin(4 * x[:, 0]))
    return vs, M.EulerSolver(*vs, conf=M.Struct(cfl=0.3, gamma=1.4))


KINDS = {"triangles": (2, lambda d: _advdiff(d, 2, "fp64"), 1e-12), "tetrahedra": (3, lambda d: _advdiff(d, 3, "fp64"), 1e-12),
         "triangles fp32c": (2, lambda d: _advdiff(d, 2, "fp32c"), 0.0),
         "tetrahedra fp32c": (3, lambda d: _advdiff(d, 3, "fp32c"), 0.0),
         "sw": (2, lambda d: _five(d, "sw"), 0.0), "euler": (2, lambda d: _five(d, "euler"), 0.0)}


@pytest.mark.parametrize("short_of", ["tables", "coefficients"])
@pytest.mark.parametrize("kind", list(KINDS))
def test_steps_without_memory_for_tables(kind, short_of, monkeypatch, cuda):
    dim, make, tol = KINDS[kind]
    if short_of == "coefficients" and kind not in ("triangles", "tetrahedra"):
        pytest.skip("no coefficients beside the tables")
    vs, S = make(_domain(dim))
    S.advance(6)
    want = [v.cell.copy() for v in vs]
    dom = _domain(dim)
    vs, S = make(dom)

    def full(*a, **k):
        raise torch.OutOfMemoryError("no memory left")
    with monkeypatch.context() as mp:
        if short_of == "tables":
            mp.setattr(DeviceMesh, "_carve", full)
        else:
            empty, n = torch.empty, (6 if dim == 2 else 8) * dom.nbcells
            mp.setattr(torch, "empty", lambda *a, **k: full() if a[:1] == (n,) else empty(*a, **k))
        S.advance(6)
    if "fp32c" in kind:
        assert S._tab32 is None
    else:
        assert S._tiles is None and getattr(S, "_tables", None) is None
    for v, a in zip(vs, want):
        assert rel_max(v.cell, a) <= tol
    _, again = make(dom)        # with memory there again, the next solver has its tables
    again.advance(1)
    assert ("fp32c" in kind and again._tab32 is not None) or ("fp32c" not in kind and again._tiles is not None)
