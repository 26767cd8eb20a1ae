"""The one-launch Euler step on tiles (mb_euler_step_tile) gives the bits of the two-launch step
(mb_euler_step_2d): meshes of fewer cells than a tile, whole tiles and some cells over.  Equal bits
need no tolerance: both round every operation as manapy's code does."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen
from manapy_b200.device import DeviceMesh
from manapy_b200.workloads import pressure_pulse

pytestmark = pytest.mark.gpu


def _solver(dom):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    for v, a in zip(vs, pressure_pulse(dom.cells.center)):
        v.cell = a
    return vs, M.EulerSolver(*vs, conf=M.Struct(cfl=0.4, gamma=1.4))


@pytest.mark.parametrize("n,tile", [(2, 32), (4, 32), (17, 34), (17, 578), (17, 576), (17, 1024), (40, 192)])
def test_tiled_step_gives_the_two_launch_bits(n, tile, monkeypatch, cuda):
    monkeypatch.setattr(DeviceMesh, "face_tile_cells", classmethod(lambda cls, c, most=None: tile))
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(n, seed=n))
    a, A = _solver(dom)
    A._setup()
    assert A._tiles is not None and A.launches_per_step() == 1
    b, B = _solver(dom)
    monkeypatch.setattr(DeviceMesh, "face_tiles", lambda self, *k: None)
    B._setup()
    assert B._tiles is None and B.launches_per_step() == 2
    for S in (A, B):
        for _ in range(3):
            S.stepper()
            S.compute_new_val()
        S.advance(7)
        S.advance(50, graph=True)
    assert A.stepper() == B.stepper() and A.time == B.time
    for x, y in zip(a, b):
        assert np.array_equal(x.cell, y.cell) and np.isfinite(x.cell).all()
