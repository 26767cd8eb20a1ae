"""advance() of equal lengths (replayed from graphs) takes the options that the solver has when it is
called: walls, order, cfl and grav changed between the calls, against single steps.  Equal bits
need no tolerance: the same launches on the same numbers."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _solver(dom, precision, order):
    r = np.random.default_rng(4)
    cc = dom.cells.center
    h = np.where(cc[:, 0] < 0.5, 2.0, 1.0)
    state = [h, 0.3 * r.standard_normal(len(h)), 0.3 * r.standard_normal(len(h)), 0.2 * h, 0.1 * cc[:, 1]]
    vs = [M.Variable(domain=dom) for _ in range(5)]
    for v, a in zip(vs, state):
        v.cell = a
    return M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                conf=M.Struct(order=order, cfl=0.3, grav=9.81, precision=precision))


@pytest.mark.parametrize("precision,order,changes", [
    ("fp64", 1, [("walls", "reflective"), ("walls", "neumann"), ("cfl", 0.2), ("grav", 5.0)]),
    ("fp64", 2, [("order", 1), ("walls", "reflective"), ("order", 2)]),
    ("fp32c", 1, [("walls", "reflective"), ("walls", "neumann"), ("cfl", 0.2), ("grav", 5.0)])])
def test_replays_take_the_options_of_their_call(precision, order, changes, cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(16, seed=3))
    whole, single = _solver(dom, precision, order), _solver(dom, precision, order)
    for name, value in [(None, None)] + changes:
        if name:
            before = whole.h.cell.copy()
            for S in (whole, single):
                setattr(S, name, value)
        for _ in range(3):              # the second and third of a length are replays
            whole.advance(8)
            for _ in range(8):
                single.advance(1)
            for k in ("h", "hu", "hv", "hc"):
                assert np.array_equal(whole.varbs[k].cell, single.varbs[k].cell), (name, k)
    assert not np.array_equal(before, whole.h.cell)
