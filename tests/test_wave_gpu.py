"""The wave kernel on cell-ordered grids against the oracle, bit for bit:
grid sides from one cell to more levels than a warp's steps in flight hold,
irregular tissues (cells without neighbours, with one and with six), chunked
launches, and the schedules that keep rows in global memory."""

import numpy as np
import pytest

from tests import network_model as N

pytestmark = pytest.mark.gpu


def _grid(n, w, seed, count=2, edges=None, schedule=0, duration=0.6):
    from dense_b200.engine import ParameterSet
    from dense_b200.tissue import default_graph, from_edges
    rng = np.random.Generator(np.random.PCG64(seed))
    off, ids = default_graph(n, w) if edges is None else from_edges(n, edges)
    out = []
    for _ in range(count):
        p = N.cases.GRID_TEMPLATE * np.exp(rng.uniform(-0.2, 0.2, size=N.cases.GRID_TEMPLATE.size))
        out.append(ParameterSet(off, ids, p, init_conc=[1.1 * p[0], p[1] / p[0]], duration=duration, schedule=schedule))
    return out


@pytest.mark.parametrize("side", [1, 2, 3, 4, 7, 8, 13, 31, 33, 48, 64])
def test_square_grids(side):
    sets = _grid(side * side, side, side, duration=0.3 if side > 40 else 0.6)
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1), N.engine_states(N.GRID, sets, 0.01, 0.1))


@pytest.mark.parametrize("n,w", [(50, 1), (77, 5), (300, 100), (600, 3)])
def test_ragged_tissues_in_chunked_launches(n, w):
    sets = _grid(n, w, n)
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1), N.engine_states(N.GRID, sets, 0.01, 0.1, chunks=2, graph=True))


@pytest.mark.parametrize("degree", [1, 2, 6])
def test_irregular_neighbours(degree):
    n = 53
    edges = [(i, (i * 7 + 3 * j + 1) % n) for i in range(n) if i % 4 for j in range(degree) if (i * 7 + 3 * j + 1) % n != i]
    sets = _grid(n, 1, degree, edges=edges)
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1), N.engine_states(N.GRID, sets, 0.01, 0.1))


@pytest.mark.parametrize("schedule", ["SCHEDULE_SHARED_NEIGHBOUR", "SCHEDULE_WAVE_GLOBAL", "SCHEDULE_GLOBAL"])
def test_other_schedules(schedule):
    from dense_b200 import engine as E
    sets = _grid(20 * 20, 20, 4)
    hinted = _grid(20 * 20, 20, 4, schedule=getattr(E, schedule))
    N.assert_same(N.oracle_states(N.GRID, sets, 0.01, 0.1), N.engine_states(N.GRID, hinted, 0.01, 0.1))


@pytest.mark.parametrize("cells", [20, 150])
def test_unordered_sets_with_delays_in_shared_rows(cells):
    from dense_b200 import engine as E
    from tests.test_step_reads_gpu import _sets
    want = N.oracle_states(N.NETWORK, _sets(cells, False, cells, duration=1.0), 0.01, 0.1)
    got = N.engine_states(N.NETWORK, _sets(cells, False, cells, duration=1.0, schedule=E.SCHEDULE_SHARED_ROWS), 0.01, 0.1)
    N.assert_same(want, got)
