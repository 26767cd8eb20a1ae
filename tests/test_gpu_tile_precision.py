"""Second-order steps with tables against the same steps in numpy's long double (64-bit mantissa) from the
mesh's vertices: no further off, on average over the cells, than the steps without tables.

No tolerance: the tables' offsets of the face centres round to the size of a cell, those of the
other steps to the size of its coordinates, which is most of their error, so about half of it is
expected."""
import numpy as np
import pytest

import manapy_b200 as M
from manapy_b200 import meshgen
from manapy_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu
STEPS, VEL = 10, (0.7, 0.4, 0.3)
L = np.longdouble


def _add(n, idx, val):
    out = np.zeros((n,) + val.shape[1:], L)
    np.add.at(out, idx, val)
    return out


def _cross(a, b):
    return np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                     a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)


def _solve(m, r):
    """m x = r by cofactors; m [n][d][d] symmetric."""
    if m.shape[1] == 2:
        x = np.stack([m[:, 1, 1] * r[:, 0] - m[:, 0, 1] * r[:, 1], m[:, 0, 0] * r[:, 1] - m[:, 0, 1] * r[:, 0]], 1)
        return x / (m[:, 0, 0] * m[:, 1, 1] - m[:, 0, 1] ** 2)[:, None]
    c = np.stack([_cross(m[:, 1], m[:, 2]), _cross(m[:, 2], m[:, 0]), _cross(m[:, 0], m[:, 1])], 1)
    return (c * r[:, None, :]).sum(2) / (m[:, 0] * c[:, 0]).sum(1)[:, None]


def _truth(A, dim, w, dt):
    """STEPS steps of pure advection with neumann sides, as manapy's scheme has them."""
    nc, nf, cf = A["nbcells"], A["nbfaces"], A["cells_faceid"][:, :dim + 1]
    X = A["nodes_vertex"][:, :dim].astype(L)
    P, Q = X[A["cells_nodeid"][:, :dim + 1]], X[A["faces_nodeid"][:, :dim]]
    cc, fc = P.sum(1) / (dim + 1), Q.sum(1) / dim
    c0, c1 = A["faces_cellid"][:, 0], A["faces_cellid"][:, 1]
    inner = c1 >= 0
    c1 = np.where(inner, c1, c0)
    if dim == 2:
        e = P[:, 1:] - P[:, :1]
        vol = np.abs(e[:, 0, 0] * e[:, 1, 1] - e[:, 0, 1] * e[:, 1, 0]) / 2
        t = Q[:, 1] - Q[:, 0]
        N = np.stack([t[:, 1], -t[:, 0]], 1)
    else:
        vol = np.abs((_cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]) * (P[:, 3] - P[:, 0])).sum(1)) / 6
        N = _cross(Q[:, 1] - Q[:, 0], Q[:, 2] - Q[:, 0]) / 2
    N = np.where(((cc[c0] - fc) * N).sum(1)[:, None] > 0, -N, N)
    n = N / np.sqrt((N * N).sum(1))[:, None]
    gc = cc[c0] + 2 * ((fc - cc[c0]) * n).sum(1)[:, None] * n       # ghosts: the centre mirrored at the face
    si, sj = np.repeat(np.arange(nc), np.diff(A["cellnid_ptr"])), A["cellnid_idx"][:A["cellnid_ptr"][-1]]
    gi, gf = np.repeat(np.arange(nc), np.diff(A["ghostnid_ptr"])), A["ghostnid_idx"][:A["ghostnid_ptr"][-1]]
    sd, gd = cc[sj] - cc[si], gc[gf] - cc[gi]
    m = _add(nc, si, sd[:, :, None] * sd[:, None, :]) + _add(nc, gi, gd[:, :, None] * gd[:, None, :])
    flux = (N * np.array(VEL[:dim]).astype(L)).sum(1)
    least = L("1e-8") if dim == 2 else L("1e-10")
    for _ in range(STEPS):
        grad = _solve(m, _add(nc, si, sd * (w[sj] - w[si])[:, None]) + _add(nc, gi, gd * (w[c0[gf]] - w[gi])[:, None]))
        hi = np.maximum(np.maximum(w[c0], w[c1])[cf].max(1), w)
        lo = np.minimum(np.minimum(w[c0], w[c1])[cf].min(1), w)
        d = ((fc[cf] - cc[:, None]) * grad[:, None]).sum(2)
        with np.errstate(all="ignore"):
            room = np.where(d > 0, (hi - w)[:, None], (lo - w)[:, None]) / d
        psi = np.where(np.abs(d) < least, L(1), np.minimum(room, L(1))).min(1)
        value = lambda c: w[c] + psi[c] * ((fc - cc[c]) * grad[c]).sum(1)  # noqa: E731
        right = np.where(inner, value(c1), w[c0])
        F = flux * np.where(flux >= 0, value(c0), right)
        rez = -_add(nc, c0, F) + _add(nc, c1[inner], F[inner])
        w = w + dt * (rez / vol)
    return w


@pytest.mark.parametrize("dim,n,sums", [(2, 24, False), (3, 7, False), (3, 7, True)])
@pytest.mark.parametrize("seed", [1, 2])
def test_no_further_off_than_without_tables(dim, n, sums, seed, monkeypatch, cuda):
    if sums:
        monkeypatch.setattr(DeviceMesh, "TET_TILED", 0)
    dom = M.Domain(dim=dim, mesh=(meshgen.square_triangles if dim == 2 else meshgen.cube_tetrahedra)(n, seed=seed))
    x = dom.cells.center
    init = np.exp(-30 * ((x[:, 0] - 0.4) ** 2 + (x[:, 1] - 0.5) ** 2)) + 0.2 * x[:, 1]
    got = {}
    for launch in ("auto", 0):
        w, *vel = (M.Variable(domain=dom) for _ in range(4))
        for v, a in zip(vel, VEL[:dim]):
            v.face = np.full(dom.nbfaces, a)
            v.interpolate_facetocell()
        w.cell = init
        S = M.AdvectionSolver(w, vel=tuple(vel), conf=M.Struct(order=2, cfl=0.5, launch=launch))
        dt = S.stepper()
        S.advance(STEPS)
        assert ((S._tables if sums else S._tiles) is not None) == (launch == "auto")
        got[launch] = w.cell.copy()
    want = _truth(dom.host_arrays, dim, init.astype(L), L(dt))
    off = {k: float(np.abs(a.astype(L) - want).mean()) for k, a in got.items()}
    assert off[0] < 1e-15           # the scheme is the same
    assert off["auto"] <= off[0], off
