"""A launch that the driver refuses (blocks that ask for more shared memory than there is) raises, and the next
call is none the worse: the refusal is not reported a second time."""
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import _lib, meshgen

pytestmark = pytest.mark.gpu


def test_the_next_call_succeeds(cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(8, seed=1))
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = 1.0
    S = M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))
    S.advance(2)
    dt = S.stepper()
    tiles, spare = S._tiles, [t.clone() for t in S._spare]
    S._tiles = type(tiles).from_buffer_copy(tiles)
    S._tiles.face_cap = 1 << 20         # 64 MB of shared memory: refused before anything runs
    with pytest.raises(_lib.MbError):
        S.advance(1)
    S._tiles = tiles
    rows = torch.empty(4 * dom.nbcells, dtype=torch.float64, device=cuda)
    _lib.call("mb_pack_rows", dom.device_mesh.struct, S.h.dev("cell").data_ptr(), rows.data_ptr(), S._stream())
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(spare, S._spare)) and S.stepper() == dt
    with pytest.raises(_lib.MbError):
        _lib.call("mb_graph_launch", None, None)
    S.advance(8)
