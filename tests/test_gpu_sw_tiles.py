"""The one-launch shallow-water step on tiles (mb_sw_step_tile) gives the bits of the two-launch
step (mb_sw_step_ex) and of its boundary fluxes: meshes of fewer cells than a tile, whole
tiles and some cells over, both walls, both orders.  Equal bits need no tolerance: the two steps
share their arithmetic, written with its rounding."""
import numpy as np
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import meshgen
from manapy_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu


def _state(cc, seed):
    r = np.random.default_rng(seed)
    x, y = cc[:, 0], cc[:, 1]
    h = np.where(x < 0.5, 2.0, 1.0) + 0.05 * r.standard_normal(len(x))
    return [h, 0.3 * r.standard_normal(len(x)), 0.3 * r.standard_normal(len(x)), 0.1 * h * (1 + y),
            0.1 * np.exp(-((x - 0.7) ** 2 + (y - 0.5) ** 2) / 0.02)]


def _solver(dom, order, walls, seed=1):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    for v, a in zip(vs, _state(dom.cells.center, seed)):
        v.cell = a
    return vs, M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                    conf=M.Struct(order=order, cfl=0.3, grav=9.81, walls=walls))


@pytest.mark.parametrize("walls", ["neumann", "reflective"])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("n,tile", [(2, 32), (4, 32), (17, 34), (17, 578), (17, 576), (17, 1024), (40, 256)])
def test_tiled_step_gives_the_two_launch_bits(n, tile, order, walls, monkeypatch, cuda):
    monkeypatch.setattr(DeviceMesh, "face_tile_cells", classmethod(lambda cls, c: tile))
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(n, seed=n))
    a, A = _solver(dom, order, walls)
    b, B = _solver(dom, order, walls)
    A._setup(), B._setup()
    assert A._tiles is not None and A.launches_per_step() == order
    B._tiles = None
    for _ in range(5):
        for S in (A, B):
            S.stepper()
            S.compute_fluxes()
            S.compute_new_val()
        assert A.dt == B.dt
        assert A.boundary_mass_flux() == B.boundary_mass_flux()
    for steps in (1, 4, 6, 6, 6):     # graphs from the second time a length is seen
        A.advance(steps)
        B.advance(steps)
    assert A.stepper() == B.stepper()
    for x, y in zip(a, b):
        assert np.array_equal(x.cell, y.cell) and np.isfinite(x.cell).all()


@pytest.mark.parametrize("precision,steps", [("fp64", 7), ("fp64", 8), ("fp64", 270), ("fp32c", 10)])
def test_replayed_lengths_continue_single_steps(precision, steps, cuda):
    """advance() of one length again and again (graph replays, odd rests between) against single steps,
    with a field written from the host and dt set by hand in between."""
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(20, seed=3))
    runs = []
    for whole in (True, False):
        vs = [M.Variable(domain=dom) for _ in range(5)]
        for v, x in zip(vs, _state(dom.cells.center, 2)):
            v.cell = x
        S = M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4],
                                 conf=M.Struct(order=1, cfl=0.3, grav=9.81, precision=precision))
        for k in range(9):
            if k == 6:
                vs[3].cell = vs[3].cell * 0.5
            for _ in range(1 if whole else steps):
                S.advance(steps if whole else 1)
        runs.append([v.cell.copy() for v in vs[:4]] + [np.array(S.stepper())])
    for x, y in zip(*runs):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("name", ["h", "Z"])
def test_arrays_at_odd_offsets(name, cuda):
    """A cell array installed 8 bytes into its storage: the steps that read it take the two-launch step."""
    import torch
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=3))
    _, A = _solver(dom, 1, "reflective")
    _, B = _solver(dom, 1, "reflective")
    t = A.varbs[name].dev("cell")
    odd = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    odd.copy_(t)
    A.varbs[name].swap_cell(odd)
    for steps in (1, 2, 8, 8, 8):
        A.advance(steps)
        B.advance(steps)
        assert A.boundary_mass_flux() == B.boundary_mass_flux()
        assert A.stepper() == B.stepper()
    for k in A.varbs:
        assert np.array_equal(A.varbs[k].cell, B.varbs[k].cell)
