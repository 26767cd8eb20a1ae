"""The one-launch step on tiles of triangles (mb_advdiff_step_tile) against the oracle, where its
tables can go wrong: meshes of fewer cells than a tile, one cell more or less than whole
tiles, every boundary rule, and vertices of many cells.

Tolerance: a step changes a value by some hundred rounded operations on numbers of its size, so
10 steps stay within 1e3 * 2^-53 ~ 1e-13 of the oracle; 1e-12 as for the other steps.
"""
import numpy as np
import pytest

from conftest import rel_max
import manapy_b200 as M
from manapy_b200 import boundary as B, geometry as G, meshgen
from manapy_b200.device import DeviceMesh
import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12
STEPS = 10
MIXED = ({"in": "dirichlet", "upper": "neumannNH", "out": "neumann", "bottom": "nonslip"}, {"in": 1.5, "upper": 0.3})
# a dirichlet side after a neumann one reads the cell array at face indices
LATE = ({"upper": "neumann", "out": "neumann", "in": "slip", "bottom": "dirichlet"}, {"bottom": 1.0})
DIRICHLET = ({s: "dirichlet" for s in ("in", "out", "upper", "bottom")},
             {"in": lambda x, y, z: 1.0 + y, "out": 0.0, "upper": 0.5, "bottom": 0.0})


def _fan(cells):
    """A disc of ``cells`` triangles around one vertex."""
    a = 2 * np.pi * np.arange(cells) / cells
    r = 1 + 0.1 * np.cos(3 * a)
    vx = np.zeros((cells + 1, 4))
    vx[1:, 0], vx[1:, 1], vx[1:, 3] = r * np.cos(a), r * np.sin(a), 1
    k = np.arange(cells)
    el = np.stack([np.zeros_like(k), 1 + k, 1 + (k + 1) % cells, np.full_like(k, 3)], 1).astype(np.int32)
    return el, vx


def _run(el, vx, bc, order, diffusion, monkeypatch=None, tile=None, seed=0):
    r = np.random.default_rng(seed)
    A = G.build(el, vx, 2)
    D = (2e-3, 1e-3, 0.0) if diffusion else (0.0, 0.0, 0.0)
    cc, fc = A["cells_center"], A["faces_center"]
    init = 1 + np.sin(3 * cc[:, 0]) * np.cos(2 * cc[:, 1]) + 0.1 * r.standard_normal(len(cc))
    vel = [np.cos(2 * fc[:, 1]), 0.5 + 0.3 * np.sin(3 * fc[:, 0]), np.zeros(len(fc))]
    src = 0.2 * r.standard_normal(len(cc))
    if tile is not None:
        monkeypatch.setattr(DeviceMesh, "tile_cells", classmethod(lambda cls, n: tile))
    dom = M.Domain(dim=2, mesh=(el, vx))
    w = M.Variable(domain=dom, BC=bc[0], values=bc[1])
    o = O.AdvDiffOracle(A, B.resolve(A, *bc), *D, order=order, cfl=0.6)
    vs = [M.Variable(domain=dom) for _ in range(3)]
    for v, a in zip(vs, vel):
        v.face = a
        v.interpolate_facetocell()
    w.cell = init
    S = M.AdvectionDiffusionSolver(w, vel=tuple(vs), conf=M.Struct(Dxx=D[0], Dyy=D[1], order=order, cfl=0.6))
    w.source = src
    o.set_velocity(*vel)
    o.w[:] = init
    o.src[:] = src
    for _ in range(STEPS):
        S.stepper()
        S.compute_fluxes()
        S.compute_new_val()
        o.step()
    return S, w, o


@pytest.mark.parametrize("order,diffusion", [(1, True), (2, True), (2, False)])
@pytest.mark.parametrize("bc", [DIRICHLET, MIXED, LATE], ids=["dirichlet", "mixed", "cell-at-face"])
@pytest.mark.parametrize("n,tile", [(2, 32), (4, 32), (17, 34), (17, 578), (17, 576), (17, 1024), (40, 384)])
def test_tiled_step_matches_oracle(n, tile, bc, order, diffusion, monkeypatch, cuda):
    """8, 32 and 578 cells: less than a tile, exactly one, 17 tiles, two cells left over, odd sizes."""
    el, vx = meshgen.square_triangles(n, seed=n)
    S, w, o = _run(el, vx, bc, order, diffusion, monkeypatch, tile)
    assert S._tiles is not None and S.launches_per_step() == 1
    assert rel_max(w.cell, o.w) < TOL


@pytest.mark.parametrize("cells,tiled", [(7, True), (101, True), (700, True), (1500, False), (5001, False)])
def test_vertices_of_many_cells(cells, tiled, cuda):
    """A vertex of 700 cells is in every tile's list; of 1500 the lists take more shared memory than two
    blocks of an SM have, of 5001 they are past the tiles' tables: the two-launch step."""
    el, vx = _fan(cells)
    bc = ({s: "dirichlet" for s in ("in", "out", "upper", "bottom")}, {s: 1.0 for s in ("in", "out", "upper", "bottom")})
    S, w, o = _run(el, vx, bc, 2, True)
    assert (S._tiles is not None) == tiled
    assert rel_max(w.cell, o.w) < TOL


def test_uniform_state_stays_exactly_uniform(cuda):
    """Gradients are sums of products of differences: a constant state has none."""
    el, vx = meshgen.square_triangles(60, seed=4)
    dom = M.Domain(dim=2, mesh=(el, vx))
    w = M.Variable(domain=dom)
    vs = [M.Variable(domain=dom) for _ in range(3)]
    w.cell = np.full(len(el), 0.7)
    S = M.AdvectionDiffusionSolver(w, vel=tuple(vs), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, order=2, cfl=0.6))
    S.advance(5, graph=False)
    assert S._tiles is not None
    assert np.array_equal(w.cell, np.full(len(el), 0.7))


@pytest.mark.parametrize("graph", [False, True])
def test_array_at_an_odd_offset(graph, cuda):
    """A cell array installed 8 bytes into its storage: the steps that read it take the two-launch step."""
    import torch
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(20, seed=4))
    out = []
    for odd in (False, True):
        w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
        w.cell = np.sin(5 * dom.cells.center[:, 0])
        u.face, v.face = np.ones(len(u.face)), np.full(len(u.face), 0.5)
        S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=2e-3, order=2, cfl=0.5,
                                                                       graph_depth=4))
        if odd:
            t = w.dev("cell")
            x = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
            x.copy_(t)
            w.swap_cell(x)
        S.advance(STEPS, graph=graph)
        out.append(w.cell.copy())
    assert rel_max(out[1], out[0]) < TOL
