"""The FP32-compensated step with its coefficients in tables (mb_advdiff_step_f32c_tab) gives the bits
of the step that forms them (mb_advdiff_step_f32c): triangles and tetrahedra, both orders, sides
with and without a diffusive gradient.  Equal bits need no tolerance: the same operations on the
same numbers, compiled without multiply-add contraction."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu
MIXED = {2: ({"in": "dirichlet", "upper": "neumannNH", "out": "neumann", "bottom": "nonslip"}, {"in": 1.5, "upper": 0.3}),
         3: ({"in": "dirichlet", "front": "neumannNH", "out": "neumann", "upper": "nonslip", "bottom": "neumann",
              "back": "slip"}, {"in": 1.5, "front": 0.3})}


def _solver(dom, dim, order, diffusion, bc):
    r = np.random.default_rng(7)
    cc, fc = dom.cells.center, dom.faces.center
    w = M.Variable(domain=dom, BC=bc[0], values=bc[1])
    vs = [M.Variable(domain=dom) for _ in range(3)]
    for v, a in zip(vs, (np.cos(2 * fc[:, 1]), 0.5 + 0.3 * np.sin(3 * fc[:, 0]), 0.2 - 0.4 * fc[:, 2] * (dim - 2))):
        v.face = a
        v.interpolate_facetocell()
    w.cell = 1 + np.sin(3 * cc[:, 0]) * np.cos(2 * cc[:, 1]) + 0.1 * r.standard_normal(len(cc))
    D = (2e-3, 1e-3, 5e-4 * (dim - 2)) if diffusion else (0.0, 0.0, 0.0)
    S = M.AdvectionDiffusionSolver(w, vel=tuple(vs), conf=M.Struct(Dxx=D[0], Dyy=D[1], Dzz=D[2], order=order, cfl=0.5,
                                                                   precision="fp32c"))
    w.source = 0.2 * r.standard_normal(len(cc))
    S._setup()
    S._f32_state()
    return w, S


@pytest.mark.parametrize("order,diffusion", [(1, True), (2, True), (2, False), (1, False)])
@pytest.mark.parametrize("dim,n", [(2, 2), (2, 17), (2, 60), (3, 2), (3, 5), (3, 9)])
def test_tables_give_the_same_bits(dim, n, order, diffusion, cuda):
    mesh = meshgen.square_triangles(n, seed=n) if dim == 2 else meshgen.cube_tetrahedra(n, seed=n)
    dom = M.Domain(dim=dim, mesh=mesh)
    a, A = _solver(dom, dim, order, diffusion, MIXED[dim])
    b, B = _solver(dom, dim, order, diffusion, MIXED[dim])
    assert A._tab32 is not None
    B._tab32 = None
    for S in (A, B):
        S.advance(5)
        S.advance(6, graph=True)
    x, y = a.cell, b.cell
    assert np.array_equal(x, y) and np.isfinite(x).all()
