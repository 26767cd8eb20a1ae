"""The FP32-compensated step with its coefficients in tables knows the faces that carry a diffusive gradient
from the mesh, not from a coefficient that happens to be zero: with D_xx = -D_yy, faces at 45 degrees
have n.D n = 0 and a tangential term.  Equal bits to the step that forms its coefficients, as
for other coefficients."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu


def _solver(dom, order):
    r = np.random.default_rng(7)
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    w.cell = 1 + 0.5 * r.random(len(w.cell))
    S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=-1e-3, order=order, precision="fp32c",
                                                                   dt=1e-3))
    S._setup()
    S._f32_state()
    return w, S


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("dim,n", [(2, 8), (3, 4)])
def test_tangential_terms_stay(dim, n, order, cuda):
    make = meshgen.square_triangles if dim == 2 else meshgen.cube_tetrahedra
    dom = M.Domain(dim=dim, mesh=make(n, seed=n, jitter=0.0))
    a, A = _solver(dom, order)
    b, B = _solver(dom, order)
    assert A._tab32 is not None
    B._tab32 = None
    for _ in range(3):
        for S in (A, B):
            S.compute_fluxes()
            S.compute_new_val()
    x, y = a.cell, b.cell
    assert np.isfinite(x).all() and np.array_equal(x, y)
