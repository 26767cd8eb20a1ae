"""After a graph replay the arrays that manapy's compute_fluxes leaves behind are those of the last step, also
when the program installed a cell array of its own since the capture.  Equal bits to a solver that
takes the same steps one by one."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before,after", [(1, 1), (1, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("dim", [2, 3])
def test_arrays_of_the_last_step(dim, before, after, cuda):
    dom = M.Domain(dim=dim, mesh=meshgen.square_triangles(10, seed=1) if dim == 2 else meshgen.cube_tetrahedra(4, seed=1))
    runs = []
    for graph in (True, False):
        w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
        u.face = 0.5
        u.interpolate_facetocell()
        w.cell = 1 + 0.2 * np.sin(5 * dom.cells.center[:, 0])
        S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, Dzz=1e-3 * (dim - 2), order=2,
                                                                       cfl=0.4, graph_depth=8))

        def steps(n, graph):
            for _ in range(1 if graph else n):
                S.advance(n if graph else 1, graph=graph)
        steps(16, graph)
        steps(before, False)
        w.swap_cell(w.dev("cell") * 1.25)
        steps(after, False)
        steps(16, graph)
        runs.append([w.cell.copy(), w.convective.copy(), w.dissipative.copy(), w.ghost.copy()])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
