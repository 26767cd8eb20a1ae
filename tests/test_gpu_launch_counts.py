"""launches_per_step() counts the launches of the step that the arrays allow: one that is installed 8 bytes
into its storage takes the two-launch step."""
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _odd(var):
    t = var.dev("cell")
    odd = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    odd.copy_(t)
    var.swap_cell(odd)


@pytest.mark.parametrize("order", [1, 2])
def test_shallow_water(order, cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(6, seed=1))
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = 1.0
    S = M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=order, cfl=0.3))
    S.advance(1)
    assert S.launches_per_step() == order
    _odd(vs[4])
    assert S.launches_per_step() == order + 1


def test_advection_diffusion(cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(6, seed=1))
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    u.face = 0.5
    u.interpolate_facetocell()
    w.cell = 1.0
    S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, order=2, cfl=0.4))
    S.advance(1)
    assert S.launches_per_step() == 1
    _odd(w)
    assert S.launches_per_step() == 2
    S.advance(2)        # to the solver's own buffer, and back to the odd one
    assert S.launches_per_step() == 2
