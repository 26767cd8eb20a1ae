"""A capture that is interrupted (a keyboard interrupt among its launches) leaves the solver where it was: the steps
were recorded, not taken.  Equal bits to a solver that was not interrupted."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import _lib, meshgen

pytestmark = pytest.mark.gpu


def _solver(dom, precision):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = np.where(dom.cells.center[:, 0] < 0.5, 2.0, 1.0)
    return M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                conf=M.Struct(order=1, cfl=0.3, precision=precision))


@pytest.mark.parametrize("at", [1, 2, 7, 16])
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_nothing_is_taken(precision, at, monkeypatch, cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(10, seed=1))
    S, other = _solver(dom, precision), _solver(dom, precision)
    S.advance(16)
    plain, seen = _lib.call, []

    def interrupted(name, *args):
        if "_step_" in name:
            seen.append(name)
            if len(seen) == at:
                raise KeyboardInterrupt
        return plain(name, *args)
    with monkeypatch.context() as mp:
        mp.setattr(_lib, "call", interrupted)
        with pytest.raises(KeyboardInterrupt):
            S.advance(16)               # the length's second time: captured
    assert not S._graphs.by_key
    for steps in (1, 16, 16, 16):
        S.advance(steps)
    for _ in range(16 + 49):
        other.advance(1)
    for k in ("h", "hu", "hv", "hc"):
        assert np.array_equal(S.varbs[k].cell, other.varbs[k].cell)
    assert S.stepper() == other.stepper()
