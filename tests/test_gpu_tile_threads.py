"""Two threads that step two solvers whose blocks take different amounts of shared memory: no launch is
refused and each gets the bits it gets alone.  The threads repeat the library call of a step, which
leaves the interpreter lock, as fast as they can."""
import threading

import numpy as np
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import _lib, meshgen
from manapy_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu
CALLS = 20000


def _advdiff(dom, dim):
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    for var, a in zip((u, v, z), (0.7, 0.4, 0.3)):
        var.face = np.full(len(var.face), a)
        var.interpolate_facetocell()
    w.cell = 1 + 0.2 * np.sin(5 * dom.cells.center[:, 0])
    return [w], M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, Dzz=1e-3 * (dim - 2),
                                                                           order=2, cfl=0.4))


def _five(dom, kind):
    vs = [M.Variable(domain=dom) for _ in range(5)]
    x = dom.cells.center
    if kind == "sw":
        vs[0].cell = np.where(x[:, 0] < 0.5, 2.0, 1.0)
        return vs[:4], M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))
    for v, a in zip(vs, (1.0, 1.0, 0.1, 0.1, 2.5)):
        v.cell = a * (1 + 0.1 * np.sin(4 * x[:, 0]))
    return vs, M.EulerSolver(*vs, conf=M.Struct(cfl=0.3, gamma=1.4))


KINDS = {   # tile sizes (both above the 48 KB that every kernel may have), the method that chooses them, mesh, solver
    "triangles": ((320, 384), "tile_cells", lambda: meshgen.square_triangles(40, seed=1), lambda d: _advdiff(d, 2)),
    "tetrahedra": ((192, 256), "tet_tile_cells", lambda: meshgen.cube_tetrahedra(9, seed=1), lambda d: _advdiff(d, 3)),
    "sw": ((384, 768), "face_tile_cells", lambda: meshgen.square_triangles(40, seed=1), lambda d: _five(d, "sw")),
    "euler": ((320, 640), "face_tile_cells", lambda: meshgen.square_triangles(40, seed=1), lambda d: _five(d, "euler"))}


@pytest.mark.parametrize("kind", list(KINDS))
def test_two_threads_step_two_tilings(kind, monkeypatch, cuda):
    sizes, chooser, mesh, make = KINDS[kind]
    calls, outs, keep = [], [], []
    for tile in sizes:
        monkeypatch.setattr(DeviceMesh, chooser, classmethod(lambda cls, n, most=None, tile=tile: tile))
        vs, S = make(M.Domain(dim=3 if kind == "tetrahedra" else 2, mesh=mesh()))
        S._setup()
        assert S._tiles is not None and S._tiles.cells == tile
        S.advance(1)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream), monkeypatch.context() as mp:
            plain, seen = _lib.call, []
            mp.setattr(_lib, "call", lambda name, *a: (seen.append((name, a)), plain(name, *a)))
            S.advance(1)        # repeated with its arguments below: it reads one set of buffers and writes another
        (name, args), = [s for s in seen if "_step_" in s[0]]
        calls.append((getattr(_lib.lib(), name), args))
        outs.append([v.dev("cell") for v in vs])
        keep.append((vs, S, stream))
    torch.cuda.synchronize()
    want = [[t.clone() for t in o] for o in outs]
    codes = [set(), set()]
    start = threading.Barrier(2)

    def run(k):
        fn, args = calls[k]
        start.wait()
        for _ in range(CALLS):
            codes[k].add(fn(*args))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{_lib.MB_OK}, {_lib.MB_OK}]
    for o, w in zip(outs, want):
        for a, b in zip(o, w):
            assert torch.equal(a, b)
