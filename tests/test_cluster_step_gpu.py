"""Tissues spread over a cluster of CTAs (register kernel) against the oracle
bit for bit: just above one CTA, at and past whole CTAs, up to the largest
cluster and one cell past it (memory kernel); one parameter row or one per
cell, every analysis, FP32 against the memory kernel, and run states that
either kernel continues from the other."""

import numpy as np
import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _analyses, _sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell", [False, True])
@pytest.mark.parametrize("cells", [257, 300, 512, 513, 733, 1024])
def test_cluster_matches_oracle(cells, per_cell):
    sets = _sets(cells, per_cell, cells, count=2, duration=1.2)
    an = _analyses(cells)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1, an), N.engine_states(N.NETWORK, sets, 0.01, 0.1, an))


@pytest.mark.parametrize("cells", [2049, 4096, 4097])
def test_largest_clusters(cells):
    sets = _sets(cells, False, cells, count=1, duration=0.3)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.1), N.engine_states(N.NETWORK, sets, 0.01, 0.1, chunks=2))


def test_many_sets_of_many_sizes():
    """More CTAs than SMs (the two-CTA variant), several cluster sizes and
    one-CTA sets in one graph."""
    rng = np.random.Generator(np.random.PCG64(5))
    sets = [_sets(int(n), False, i, count=1, duration=0.5)[0]
            for i, n in enumerate(rng.integers(30, 1100, size=90))]
    got = N.engine_states(N.NETWORK, sets, 0.01, 0.1, graph=True)
    pick = list(range(0, 90, 9))
    N.assert_same(N.oracle_states(N.NETWORK, [sets[i] for i in pick], 0.01, 0.1), [got[i] for i in pick])


@pytest.mark.parametrize("precision", [0, 1])
def test_checks_drop_the_set_in_every_cta(precision):
    """A concentration check that one cell of the last CTA fails."""
    from dense_b200 import engine as E
    def run(schedule):
        sets = _sets(600, True, 3, count=3, duration=2.0, schedule=schedule)
        sets[1].cell_params[590, 0] *= 40.0  # its m0 runs away
        an = [E.Analysis.conccheck([0], 0, 600, -1.0, 120.0), E.Analysis.basic([0], 0, 600)]
        return N.engine_states(N.NETWORK, sets, 0.01, 0.1, an, precision=precision)
    got, want = run(E.SCHEDULE_AUTO), run(E.SCHEDULE_MEMORY)
    assert got[1]["status"] & E.SET_DROPPED and not got[0]["status"] & E.SET_DROPPED
    for g, w in zip(got, want):
        assert g["status"] == w["status"]
        for k in w[1]:
            assert np.array_equal(g[1][k], w[1][k]), k
        assert np.array_equal(g["state"], w["state"])


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_run_states_pass_between_the_kernels(order):
    from dense_b200 import engine as E
    hints = (E.SCHEDULE_AUTO, E.SCHEDULE_MEMORY)
    mk = lambda schedule: _sets(420, False, 8, count=2, duration=1.0, schedule=schedule)  # noqa: E731
    lib = N.engine_library(N.NETWORK)
    a = E.Batch(lib, mk(hints[order[0]]), 0.01, 0.1, _analyses(420))
    a.run(4)
    snap = a.checkpoint()
    a.close()
    b = E.Batch(lib, mk(hints[order[1]]), 0.01, 0.1, _analyses(420))
    b.restore(snap)
    b.run()
    b.sync()
    got = [{"state": b.state(i), 0: b.basic(0, i), 1: b.oscillation(1, i)} for i in range(2)]
    b.close()
    N.assert_same(N.oracle_states(N.NETWORK, mk(0), 0.01, 0.1, _analyses(420)), got)
