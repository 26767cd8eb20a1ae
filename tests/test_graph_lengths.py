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
