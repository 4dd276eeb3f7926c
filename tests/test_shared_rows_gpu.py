"""The wave kernel on unordered sets (rows in shared memory on request), whose
row counters advance step by step: rows of every depth, one to four steps in
flight, runs cut into launches with and without analyses, against the oracle
bit for bit."""

import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _analyses, _sets
from tests.test_wave_gpu import _grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [None, 1, 3])
@pytest.mark.parametrize("cells,per_cell", [(1, False), (40, False), (200, True), (500, False)])
@pytest.mark.parametrize("analyses", [False, True])
def test_unordered_sets(cells, per_cell, chunks, analyses):
    from dense_b200 import engine as E
    an = _analyses(cells) if analyses else []
    mk = lambda s: _sets(cells, per_cell, 3, count=2, duration=0.7, schedule=s)  # noqa: E731
    N.assert_same(N.oracle_states(N.NETWORK, mk(0), 0.01, 0.1, an),
                  N.engine_states(N.NETWORK, mk(E.SCHEDULE_SHARED_ROWS), 0.01, 0.1, an, chunks=chunks))


@pytest.mark.parametrize("chunks", [None, 1, 3])
@pytest.mark.parametrize("block", [0, 32, 64, 128])
def test_steps_in_flight(block, chunks):
    sets = _grid(81, 9, 4, duration=0.7)
    want = N.oracle_states(N.GRID, sets, 0.01, 0.1)
    for s in sets:
        s.mem_block = block
    N.assert_same(want, N.engine_states(N.GRID, sets, 0.01, 0.1, chunks=chunks))
