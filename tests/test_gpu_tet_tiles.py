"""The second-order steps on tetrahedra, on tiles (mb_advdiff_step_tet) and with the sums in memory
(mb_advdiff_step_tet_sums), against the oracle: meshes of fewer cells than a tile, whole tiles and
some cells over, sides of several kinds, with and without diffusion.

Tolerance: a step changes a value by some hundred rounded operations on numbers of its size, so 8
steps stay within 1e3 * 2^-53 ~ 1e-13 of the oracle; 1e-12 as for the other steps.
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
STEPS = 8
SIDES = ("in", "out", "upper", "bottom", "front", "back")
DIRICHLET = ({s: "dirichlet" for s in SIDES}, {s: (1.0 if s == "in" else 0.2) for s in SIDES})
MIXED = ({"in": "dirichlet", "out": "neumann", "upper": "nonslip", "bottom": "neumann", "front": "slip",
          "back": "nonslip"}, {"in": 1.5})


def _run(n, bc, diffusion, seed=0):
    r = np.random.default_rng(seed)
    el, vx = meshgen.cube_tetrahedra(n, seed=n)
    A = G.build(el, vx, 3)
    D = (2e-3, 1e-3, 5e-4) if diffusion else (0.0, 0.0, 0.0)
    cc, fc = A["cells_center"], A["faces_center"]
    init = 1 + np.sin(3 * cc[:, 0]) * np.cos(2 * cc[:, 1]) + 0.1 * r.standard_normal(len(cc))
    vel = [np.cos(2 * fc[:, 1]), 0.5 + 0.3 * np.sin(3 * fc[:, 0]), 0.2 - 0.4 * fc[:, 2]]
    src = 0.2 * r.standard_normal(len(cc))
    dom = M.Domain(dim=3, mesh=(el, vx))
    w = M.Variable(domain=dom, BC=bc[0], values=bc[1])
    o = O.AdvDiffOracle(A, B.resolve(A, *bc), *D, order=2, cfl=0.6)
    vs = [M.Variable(domain=dom) for _ in range(3)]
    for v, a in zip(vs, vel):
        v.face = a
        v.interpolate_facetocell()
    w.cell = init
    S = M.AdvectionDiffusionSolver(w, vel=tuple(vs), conf=M.Struct(Dxx=D[0], Dyy=D[1], Dzz=D[2], order=2, cfl=0.6))
    w.source = src
    o.set_velocity(*vel)
    o.w[:] = init
    o.src[:] = src
    S.advance(3)
    S.advance(STEPS - 3, graph=True)
    for _ in range(STEPS):
        o.step()
    return S, w, o


@pytest.mark.parametrize("diffusion", [True, False])
@pytest.mark.parametrize("bc", [DIRICHLET, MIXED], ids=["dirichlet", "mixed"])
@pytest.mark.parametrize("n,tile", [(2, 32), (2, 48), (2, 96), (4, 32), (5, 62), (5, 256), (7, 128)])
def test_tiled_step_matches_oracle(n, tile, bc, diffusion, monkeypatch, cuda):
    """48, 384, 750 and 2058 cells: a tile and a half, exactly one, less than one, many, a ragged end."""
    monkeypatch.setattr(DeviceMesh, "tet_tile_cells", classmethod(lambda cls, c: tile))
    S, w, o = _run(n, bc, diffusion)
    assert S._tiles is not None and S.launches_per_step() == 2
    assert rel_max(w.cell, o.w) < TOL


@pytest.mark.parametrize("diffusion", [True, False])
@pytest.mark.parametrize("bc", [DIRICHLET, MIXED], ids=["dirichlet", "mixed"])
@pytest.mark.parametrize("n", [2, 5, 7])
def test_step_with_sums_in_memory_matches_oracle(n, bc, diffusion, monkeypatch, cuda):
    monkeypatch.setattr(DeviceMesh, "TET_TILED", 0)
    S, w, o = _run(n, bc, diffusion)
    assert S._tiles is None and S._tables is not None and S.launches_per_step() == 3
    assert rel_max(w.cell, o.w) < TOL
