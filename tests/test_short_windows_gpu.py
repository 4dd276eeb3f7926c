"""Oscillation windows whose middle slot is dequeued before it is looked at --
one, three and five samples, and windows that the run is too short for or that
species late in a list hardly fill -- against the oracle bit for bit, in each
kernel that samples."""

import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from tests.test_wave_gpu import _grid

pytestmark = pytest.mark.gpu
INF = float("inf")


def _osc(species, cells, window):
    from dense_b200.engine import Analysis
    return Analysis.oscillation(species, 0, cells, 0.0, INF, window, 0.1)


@pytest.mark.parametrize("window", [0.05, 0.1, 0.2, 0.35, 0.45, 0.55, 0.65, 0.75, 0.95, 1.05])
@pytest.mark.parametrize("chunks", [None, 1, 7])
def test_windows(window, chunks):
    sets = _sets(37, False, 4, duration=3.0)
    an = [_osc([3, 8, 13, 4, 9], 37, window), _osc([0, 5], 37, window)]
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1, an),
                  N.engine_states(N.NETWORK, sets, 0.01, 0.1, an, chunks=chunks))


@pytest.mark.parametrize("samples", [1, 2, 3, 4, 5, 6, 9, 10])
@pytest.mark.parametrize("window", [0.15, 0.35, 0.45, 0.65, 1.05, 2.05])
def test_runs_shorter_than_the_window(window, samples):
    sets = _sets(20, False, 4, duration=0.1 * samples - 0.05)
    an = [_osc(list(range(14)), 20, window)]
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1, an), N.engine_states(N.NETWORK, sets, 0.01, 0.1, an))


@pytest.mark.parametrize("window", [0.35, 0.55])
@pytest.mark.parametrize("cells,schedule", [(200, "SCHEDULE_MEMORY"), (300, "SCHEDULE_AUTO"), (200, "SCHEDULE_AUTO")])
def test_kernels(cells, schedule, window):
    from dense_b200 import engine as E
    an = [_osc([0, 5, 13], cells, window)]
    N.assert_same(N.oracle_states(N.NETWORK, _sets(cells, False, 6), 0.01, 0.1, an),
                  N.engine_states(N.NETWORK, _sets(cells, False, 6, schedule=getattr(E, schedule)), 0.01, 0.1, an))


@pytest.mark.parametrize("window", [0.1, 0.35, 0.55])
def test_wave_kernel(window):
    an = [_osc([1, 0], 100, window)]
    sets = _grid(100, 10, 3, duration=2.0)
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1, an), N.engine_states(N.GRID, sets, 0.01, 0.1, an))
