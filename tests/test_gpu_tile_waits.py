"""A step on tiles whose copies do not arrive reports it in a word that the solver's next calls raise on.
The wait that runs out here is one for copies that were never issued, with a short limit; the
kernel returns and the context stays usable."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT
import manapy_b200 as M
from manapy_b200 import _lib, meshgen


def test_tile_structs_match_the_header(tmp_path):
    structs = {"mb_tiles": _lib.MbTiles, "mb_tet_tiles": _lib.MbTetTiles, "mb_face_tiles": _lib.MbFaceTiles}
    lines = ['#include <stdio.h>', '#include <stddef.h>', '#include "manapy_b200.h"', "int main(void) {"]
    for name, cls in structs.items():
        lines.append('printf("%%zu", sizeof(%s));' % name)
        lines += ['printf(" %%zu", offsetof(%s, %s));' % (name, field) for field, _ in cls._fields_]
        lines.append('printf("\\n");')
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines + ["return 0; }"]))
    exe = str(tmp_path / "layout")
    subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", exe], check=True)
    rows = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    for row, cls in zip(rows, structs.values()):
        assert [int(x) for x in row.split()] == [ctypes.sizeof(cls)] + [getattr(cls, f).offset for f, _ in cls._fields_]


def _expire(word):
    _lib.call("mb_tile_wait_check", 2, word.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [True, False])
def test_a_wait_that_runs_out_is_reported(pinned, cuda):
    word = torch.zeros(1, dtype=torch.int32, pin_memory=True) if pinned else torch.zeros(1, dtype=torch.int32, device=cuda)
    for limit in (0, -1, 4097):
        with pytest.raises(_lib.MbError):
            _lib.call("mb_tile_wait_check", limit, word.data_ptr(), None)
    assert int(word[0]) == 0
    _expire(word)
    assert int(word[0]) == 1
    assert float(torch.ones(1000, device=cuda).sum()) == 1000.0


def _solver(kind):
    dim = 3 if kind == "tetrahedra" else 2
    dom = M.Domain(dim=dim, mesh=meshgen.cube_tetrahedra(4, seed=1) if dim == 3 else meshgen.square_triangles(12, seed=1))
    if kind == "sw":
        vs = [M.Variable(domain=dom) for _ in range(5)]
        vs[0].cell = 1.0
        return M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))
    if kind == "euler":
        vs = [M.Variable(domain=dom) for _ in range(5)]
        for v, a in zip(vs, (1.0, 1.0, 0.1, 0.1, 2.51)):
            v.cell = a
        return M.EulerSolver(*vs, conf=M.Struct(cfl=0.3, gamma=1.4))
    w, u, v, z = (M.Variable(domain=dom) for _ in range(4))
    u.face = np.full(len(u.face), 0.7)
    u.interpolate_facetocell()
    return M.AdvectionDiffusionSolver(w, vel=(u, v, z), conf=M.Struct(Dxx=1e-3, Dyy=1e-3, order=2, cfl=0.4))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["triangles", "tetrahedra", "sw", "euler"])
def test_the_solver_raises(kind, cuda):
    S, other = _solver(kind), _solver(kind)
    for s in (S, other):
        s.stepper()
        s.advance(3)
        s.check()
        assert s._tiles.late
    _expire(S._watch.word)
    for call in (S.check, S.stepper, lambda: S.advance(1), S.compute_fluxes, S.compute_new_val):
        with pytest.raises(_lib.MbError, match="waited in vain"):
            call()
    other.advance(1)        # its word is its own
    other.check()
