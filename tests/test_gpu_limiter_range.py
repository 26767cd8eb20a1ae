"""The second-order steps limit states of any size alike: a step of values near 1e168 (2^560) is the step
of the same values near 1e18, times a power of two.

Tolerance: scaling by a power of two is exact, so both runs take the same roundings except where the
limiter finds its smallest bound by dividing instead of multiplying across: one rounding of a
face's offset, which is at most the range of the values around it.  Five steps of that, and what
they carry on, stay within 100 * 2^-53 ~ 1e-14 of the largest value.  An unlimited face is off
by 1e-2 and more."""
import numpy as np
import pytest

from conftest import rel_max
import manapy_b200 as M
from manapy_b200 import meshgen
from manapy_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu


def _run(dom, dim, exponent, diffusion):
    r = np.random.default_rng(8)
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    for var, a in zip((u, v, z), (0.7, 0.4, 0.3 * (dim - 2))):
        var.face = np.full(len(var.face), a)
        var.interpolate_facetocell()
    w.cell = np.ldexp(1 + r.random(len(w.cell)), exponent)
    D = (1e-4, 2e-4, 1e-4 * (dim - 2)) if diffusion else (0., 0., 0.)
    S = M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=D[0], Dyy=D[1], Dzz=D[2], order=2, cfl=0.5))
    S.advance(5)
    return np.ldexp(w.cell, -exponent), S


@pytest.mark.parametrize("diffusion", [True, False])
@pytest.mark.parametrize("dim,n,sums", [(2, 3, False), (2, 24, False), (3, 2, False), (3, 6, False), (3, 6, True)])
def test_large_values_are_limited_as_others(dim, n, sums, diffusion, monkeypatch, cuda):
    if sums:
        monkeypatch.setattr(DeviceMesh, "TET_TILED", 0)
    dom = M.Domain(dim=dim, mesh=meshgen.square_triangles(n, seed=n) if dim == 2 else meshgen.cube_tetrahedra(n, seed=n))
    want, A = _run(dom, dim, 60, diffusion)
    got, B = _run(dom, dim, 560, diffusion)
    assert (A._tables if sums else A._tiles) is not None
    assert np.isfinite(got).all() and rel_max(got, want) < 1e-14
