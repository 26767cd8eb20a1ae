"""Solvers of two threads that capture their graphs at the same time."""
import threading

import numpy as np
import pytest
import torch

import manapy_b200 as M
from manapy_b200 import meshgen

pytestmark = pytest.mark.gpu
ROUNDS = 60


def test_two_threads_capture(cuda):
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=2))

    def solver():
        vs = [M.Variable(domain=dom) for _ in range(5)]
        vs[0].cell = np.where(dom.cells.center[:, 0] < 0.5, 2.0, 1.0)
        return M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))

    ref = solver()
    for _ in range(2 * ROUNDS * 8):
        ref.advance(1)
    want = ref.h.cell.copy()
    solvers, errors = [solver() for _ in range(2)], []
    for S in solvers:
        S.stepper()
    torch.cuda.synchronize()
    start = threading.Barrier(2)

    def run(S):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(ROUNDS):
                    S.release_graphs()
                    S.advance(8)
                    S.advance(8)             # captured
                torch.cuda.current_stream().synchronize()
        except Exception as e:               # noqa: BLE001  (shown by the test's own thread)
            errors.append(e)

    threads = [threading.Thread(target=run, args=(S,)) for S in solvers]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for S in solvers:
        assert np.array_equal(S.h.cell, want)


def test_freeing_graphs_leaves_a_capture_alone(cuda):
    """A solver's graphs are freed while the program captures a graph of its own."""
    dom = M.Domain(dim=2, mesh=meshgen.square_triangles(12, seed=2))
    vs = [M.Variable(domain=dom) for _ in range(5)]
    vs[0].cell = 1.0
    S = M.ShallowWaterSolver(vs[0], hvel=(vs[1], vs[2]), hc=vs[3], Z=vs[4], conf=M.Struct(order=1, cfl=0.3))
    for _ in range(3):
        S.advance(8)
    x = torch.zeros(8, device=cuda)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        S.release_graphs()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 16.0
