"""advance(graph=True) of the Euler solver takes the cfl and gamma that the solver has when it is called: against
single steps, equal bits (the same launches on the same numbers)."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _solver(dom):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    x = dom.cells.center
    for v, a in zip(vs, (1.0, 1.0, 0.1, 0.1, 2.51)):
        v.cell = a * (1 + 0.1 * np.sin(4 * x[:, 0]))
    return vs, M.EulerSolver(*vs, conf=M.Struct(cfl=0.3, gamma=1.4))


def test_replays_take_the_options_of_their_call(cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=3))
    (a, whole), (b, single) = _solver(dom), _solver(dom)
    n = 2 * whole.GRAPH_DEPTH
    for name, value in (("cfl", 0.3), ("cfl", 0.15), ("gamma", 1.3), ("cfl", 0.3), ("gamma", 1.4)):
        setattr(whole, name, value)
        setattr(single, name, value)
        whole.advance(n, graph=True)
        single.advance(n)
        for x, y in zip(a, b):
            assert np.array_equal(x.cell, y.cell), (name, value)
    assert whole.time == single.time
