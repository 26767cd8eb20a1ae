"""Solvers' graph captures while garbage collections free other solvers and their graphs."""
import gc

import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _shallow_water(dom):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = np.where(dom.cells.center[:, 0] < 0.5, 2.0, 1.0)
    return vs, M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))


def test_captures_survive_garbage_collections(cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=1))
    _, ref = _shallow_water(dom)
    for _ in range(3):
        for _ in range(16):
            ref.advance(1)
    want = ref.h.cell.copy()
    old = gc.get_threshold()
    gc.set_threshold(30, 2, 2)        # collections inside the captures
    try:
        for _ in range(20):
            _, S = _shallow_water(dom)
            for _ in range(3):
                S.advance(16)         # captured the second time
            assert np.array_equal(S.h.cell, want)
            S.cycle = S               # freed by a collection only
    finally:
        gc.set_threshold(*old)
