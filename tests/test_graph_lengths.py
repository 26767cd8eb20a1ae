"""Which runs of steps the solvers capture into graphs: lengths that come back while their graph would be
kept, and no others, since a capture costs what launching its steps does."""
import pytest

from manapy_b200.solvers import _Graphs


class _Recorded(_Graphs):
    """As the solvers use it, with the graph itself left out."""

    def __init__(self):
        super().__init__()
        self.captures = self.hits = 0

    def run(self, key):
        if self.get(key) is not None:
            self.hits += 1
        elif self.worth(key):
            self.captures += 1
            self.keep(key, object())


@pytest.mark.parametrize("lengths", range(1, _Graphs.MOST + 1))
def test_lengths_that_fit_are_captured_once(lengths):
    g = _Recorded()
    for _ in range(10):
        for key in range(lengths):
            g.run(key)
    assert g.captures == lengths and g.hits == 8 * lengths


@pytest.mark.parametrize("lengths", [_Graphs.MOST + 1, _Graphs.MOST + 2, 2 * _Graphs.MOST, 3 * _Graphs.MOST])
def test_more_lengths_than_graphs_are_not_captured_again_and_again(lengths):
    g = _Recorded()
    for _ in range(10):
        for key in range(lengths):
            g.run(key)
    assert g.captures == 0


@pytest.mark.parametrize("kept", range(_Graphs.MOST + 1))
def test_kept_graphs_stay_while_too_many_lengths_come(kept):
    """Lengths captured earlier go on being replayed, and the others beside them are launched."""
    g, lengths = _Recorded(), _Graphs.MOST + 2
    for _ in range(2):
        for key in range(kept):
            g.run(key)
    assert g.captures == kept
    for _ in range(10):
        for key in range(lengths):
            g.run(key)
    assert g.captures == kept and g.hits == 10 * kept


@pytest.mark.parametrize("steps,asks", [(2, 8), (4, 4), (6, 3), (8, 2), (16, 1), (128, 1)])
def test_short_runs_pay_for_their_capture_first(steps, asks):
    """A capture costs what launching 16 steps does: as many are launched before it."""
    g = _Graphs()
    assert [g.worth("key", steps) for _ in range(asks + 1)] == [False] * asks + [True]
