"""The steps on tiles keep to the cells around a cell: a NaN or an outlier in one cell of a tile changes
the same cells after a step as in the step without tiles, and no others.

Tolerance: the cells that the outlier does not reach hold values of about 1, from some hundred rounded
operations on values of at most a few times that: 1e3 * 2^-53 ~ 1e-13; 1e-12 as for the other steps.
"""
import numpy as np
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu
MESHES = {2: lambda: meshgen.square_triangles(24, seed=5), 3: lambda: meshgen.cube_tetrahedra(6, seed=5)}
SIDES = {2: ("in", "out", "upper", "bottom"), 3: ("in", "out", "upper", "bottom", "front", "back")}


def _step(dom, launch, at, value):
    w = M.Variable(domain=dom, BC={s: "dirichlet" for s in SIDES[dom.dim]}, values={s: 1.0 for s in SIDES[dom.dim]})
    u, v, z = (M.Variable(domain=dom) for _ in range(3))
    for var, a in zip((u, v, z), (0.7, 0.4, 0.3)):
        var.face = np.full(len(var.face), a)
        var.interpolate_facetocell()
    x = dom.cells.center
    w.cell = 1 + 0.2 * np.sin(5 * x[:, 0]) * np.cos(4 * x[:, 1])
    S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=2e-3, Dzz=1e-3, order=2, cfl=0.4,
                                                                   launch=launch))
    t = w.dev("cell").clone()
    t[at] = value
    w.swap_cell(t)
    S.advance(1)
    assert (S._tiles is not None) == (launch == "auto")
    return w.dev("cell").cpu().numpy().copy()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("where", ["first", "last", "middle"])
def test_one_cell_reaches_the_same_cells(dim, where, cuda):
    dom = M.Domain(dim=dim, mesh=MESHES[dim]())
    dm = dom.device_mesh
    tile = dm.tile_cells(dm.nbcells) if dim == 2 else dm.tet_tile_cells(dm.nbcells)
    at = {"first": 2 * tile, "last": 3 * tile - 1, "middle": 4 * tile + tile // 2}[where]
    plain = _step(dom, 0, at, torch.nan)
    tiled = _step(dom, "auto", at, torch.nan)
    assert np.isnan(plain).any() and not np.isnan(plain).all()
    assert np.array_equal(np.isnan(tiled), np.isnan(plain))
    ok = ~np.isnan(plain)
    assert np.max(np.abs(tiled[ok] - plain[ok])) < 1e-12
    far = _step(dom, "auto", at, 1e9)        # the cells a NaN does not reach
    assert np.max(np.abs(far[ok] - plain[ok])) < 1e-12
