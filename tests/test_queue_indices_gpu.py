"""The analyses' state across samples, against the oracle bit for bit: window
sizes (even numbers of samples) up to longer than the run, several analyses
with ranges of cells and times of their own, species counts around those that
a thread loads at once, runs cut into launches, in each kernel that samples."""

import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from tests.test_wave_gpu import _grid

pytestmark = pytest.mark.gpu


def _some(cells, species, window):
    from dense_b200.engine import Analysis
    inf = float("inf")
    order = [(5 * i + 3) % len(N.cases.NETWORK_SPECIES) for i in range(species)]
    return [Analysis.oscillation(order, 0, cells, 0.0, inf, window, 0.1),
            Analysis.basic(order, 0, cells),
            Analysis.oscillation([0, 5, 13], cells // 3, cells, 0.35, 2.05, 0.4, 0.1),
            Analysis.basic([13], cells // 2, cells, 0.55, 1.25)]


@pytest.mark.parametrize("window", [0.2, 0.3, 0.8, 9.0])
@pytest.mark.parametrize("chunks", [None, 1, 7])
def test_register_kernel(window, chunks):
    sets = _sets(37, False, 4, duration=3.0)
    an = _some(37, 5, window)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1, an),
                  N.engine_states(N.NETWORK, sets, 0.01, 0.1, an, chunks=chunks))


@pytest.mark.parametrize("species", [1, 3, 4, 7, 14])
@pytest.mark.parametrize("cells,count", [(1, 2), (15, 2), (17, 160), (300, 2)])
def test_species_counts(cells, count, species):
    sets = _sets(cells, cells == 300, species, count=count, duration=1.0)
    an = [_some(cells, min(species, 7), 0.4)[0], _some(cells, species, 0.4)[1]]
    got = N.engine_states(N.NETWORK, sets, 0.01, 0.1, an, chunks=4, graph=True)
    N.assert_same(N.oracle_states(N.NETWORK, sets[:4], 0.01, 0.1, an), got[:4])


@pytest.mark.parametrize("chunks", [None, 3])
@pytest.mark.parametrize("schedule", ["SCHEDULE_MEMORY", "SCHEDULE_REGISTER"])
def test_hinted_kernels(schedule, chunks):
    from dense_b200 import engine as E
    an = _some(90, 4, 0.8)
    mk = lambda s: _sets(90, False, 6, duration=2.0, schedule=s)  # noqa: E731
    N.assert_same(N.oracle_states(N.NETWORK, mk(0), 0.01, 0.1, an),
                  N.engine_states(N.NETWORK, mk(getattr(E, schedule)), 0.01, 0.1, an, chunks=chunks))


@pytest.mark.parametrize("chunks", [None, 3])
def test_wave_kernel(chunks):
    from dense_b200.engine import Analysis
    an = [Analysis.oscillation([1, 0], 0, 100, 0.0, float("inf"), 0.8, 0.1), Analysis.basic([0, 1], 5, 77),
          Analysis.oscillation([0], 11, 90, 0.25, 1.5, 0.4, 0.1)]
    sets = _grid(100, 10, 3, duration=2.0)
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1, an),
                  N.engine_states(N.GRID, sets, 0.01, 0.1, an, chunks=chunks))


def test_more_analyses_than_shared_indices():
    """Seven equal analyses of thirteen species: the fields of the last ones
    are read and written at each sample."""
    from dense_b200 import engine as E
    an = [E.Analysis.oscillation(list(range(13)), 0, 50, 0.0, float("inf"), 0.4, 0.1) for _ in range(7)]
    sets = _sets(50, False, 12, count=2, duration=2.0)
    got = N.engine_states(N.NETWORK, sets, 0.01, 0.1, an, chunks=6)
    for g in got:
        for k in range(1, 7):
            N.assert_same([{"": g[0]}], [{"": g[k]}])
