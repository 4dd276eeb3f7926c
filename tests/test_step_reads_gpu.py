"""The register kernel's resolved reads against the oracle and against the
memory kernel, bit for bit, where they can go wrong: one cell, partial and
full warps and CTAs, one parameter row or one per cell, cells with no, few
and more than six neighbours, delays of lag 0 and of DENSE's whole ring, and
delays that DENSE would read out of bounds with (flagged)."""

import numpy as np
import pytest

from tests import network_model as N

pytestmark = pytest.mark.gpu


def _sets(cells, per_cell, seed, count=3, delays=None, width=4, edges=None, duration=2.0, schedule=0, perturb=None):
    from dense_b200.engine import ParameterSet
    from dense_b200.tissue import default_graph, from_edges
    rng = np.random.Generator(np.random.PCG64(seed))
    off, ids = default_graph(cells, width) if edges is None else from_edges(cells, edges)
    p0 = N.cases._network_template()
    first = len(N.cases.NETWORK_REACTIONS)
    out = []
    for _ in range(count):
        p = p0 * np.exp(rng.uniform(-0.6, 0.6, size=p0.size))
        if delays is not None:
            p[first:first + len(N.cases.NETWORK_DELAYED)] = rng.choice(delays, size=len(N.cases.NETWORK_DELAYED))
        cell = p[None, :] * rng.uniform(0.9, 1.1, size=(cells, p.size)) if per_cell else None
        out.append(ParameterSet(off, ids, p, cell_params=cell, duration=duration, schedule=schedule, perturb=perturb,
                                init_conc=rng.uniform(0.0, 50.0, size=len(N.cases.NETWORK_SPECIES))))
    return out


def _analyses(cells):
    from dense_b200.engine import Analysis
    return [Analysis.basic([0, 13], 0, cells), Analysis.oscillation([0, 5], 0, cells, 0.0, float("inf"), 0.8, 0.1)]


@pytest.mark.parametrize("per_cell", [False, True])
@pytest.mark.parametrize("cells", [1, 2, 32, 33, 224, 225, 256])
def test_register_kernel_matches_oracle(cells, per_cell):
    sets = _sets(cells, per_cell, 10 + cells)
    an = _analyses(cells)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1, an), N.engine_states(N.NETWORK, sets, 0.01, 0.1, an))


@pytest.mark.parametrize("per_cell", [False, True])
def test_more_sets_than_one_wave(per_cell):
    """Two CTAs per SM (another variant of the kernel), in launches of a few
    chunks."""
    sets = _sets(40, per_cell, 5, count=160, duration=1.0)
    got = N.engine_states(N.NETWORK, sets, 0.01, 0.1, chunks=3)
    pick = list(range(0, 160, 16))
    N.assert_same(N.oracle_states(N.NETWORK, [sets[i] for i in pick], 0.01, 0.1), [got[i] for i in pick])


@pytest.mark.parametrize("degree", [0, 1, 3, 6, 7, 12])
@pytest.mark.parametrize("per_cell", [False, True])
def test_neighbour_counts(degree, per_cell):
    """Every third cell has no neighbours, the others `degree`."""
    n = 45
    edges = [(i, (i + 1 + 2 * j) % n) for i in range(n) if i % 3 for j in range(degree)]
    sets = _sets(n, per_cell, degree, edges=edges)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1), N.engine_states(N.NETWORK, sets, 0.01, 0.1))


@pytest.mark.parametrize("per_cell", [False, True])
@pytest.mark.parametrize("delays", [[1.0], [1.0, 2.0, 9.5], [31.5], [32.5], [0.5, 3.0]])
def test_delays_at_the_edges(delays, per_cell):
    """Lag 0, staged depths at a power of two and one past it, and (a delay
    below one at a step of one minute) the last row of DENSE's ring."""
    sets = _sets(36, per_cell, 77, delays=delays, duration=40.0)
    if per_cell:
        for s in sets:  # the same delays in every cell: only the rates vary
            first = len(N.cases.NETWORK_REACTIONS)
            s.cell_params[:, first:first + len(N.cases.NETWORK_DELAYED)] = \
                s.set_params[first:first + len(N.cases.NETWORK_DELAYED)]
    dt, interval = (1.0, 4.0) if 0.5 in delays else (0.5, 2.0)
    N.assert_same(N.oracle_states(N.NETWORK, sets, dt, interval), N.engine_states(N.NETWORK, sets, dt, interval))


@pytest.mark.parametrize("per_cell", [False, True])
def test_flagged_reads_run_the_checked_rules(per_cell):
    """Perturbation factors that shrink DENSE's rings below the delays: the
    status words and the states are the memory kernel's."""
    from dense_b200 import engine as E
    factors = np.full(len(N.cases.NETWORK_REACTIONS), -0.75)
    mk = lambda schedule: _sets(30, per_cell, 3, delays=[2.0, 7.0, 15.0], duration=30.0, perturb=factors,  # noqa: E731
                                schedule=schedule)
    got = N.engine_states(N.NETWORK, mk(E.SCHEDULE_AUTO), 1.0, 3.0)
    want = N.engine_states(N.NETWORK, mk(E.SCHEDULE_MEMORY), 1.0, 3.0)
    assert any(r["status"] & E.SET_BAD_DELAY for r in got)
    N.assert_same(want, got)
