"""advance() inside a program's own graph capture launches its steps there, also when the solver keeps graphs
of that length: replaying the program's graph gives the bits of calling advance()."""
import numpy as np
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _sw(dom, precision):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = np.where(dom.cells.center[:, 0] < 0.5, 2.0, 1.0)
    return vs[0], M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                       conf=M.Struct(order=1, cfl=0.3, precision=precision))


def _advdiff(dom, precision):
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    u.face = np.full(len(u.face), 0.7)
    u.interpolate_facetocell()
    w.cell = 1 + 0.2 * np.sin(5 * dom.cells.center[:, 0])
    return w, M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, order=2, cfl=0.4,
                                                                         precision=precision, graph_depth=16))


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("kind", ["sw", "advdiff"])
def test_advance_inside_a_capture(kind, precision, cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=2))
    a, A = (_sw if kind == "sw" else _advdiff)(dom, precision)
    b, B = (_sw if kind == "sw" else _advdiff)(dom, precision)
    extra = {} if kind == "sw" else {"graph": True}
    side = torch.cuda.Stream()
    for _ in range(3):                       # the solver has a graph of 8 steps from here on
        for S in (A, B):
            S.stepper()
            S.advance(8, **extra)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):   # 8 steps end in the buffers where they began
        A.advance(8, **extra)
    for _ in range(2):
        g.replay()
        B.advance(8, **extra)
    torch.cuda.synchronize()
    assert np.array_equal(a.cell, b.cell)
