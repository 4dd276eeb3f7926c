"""History reads with a whole number for the delay (their row is not known
before the rates run) and delayed reads behind a condition on such a read, in
the register kernel against the oracle bit for bit; and a delayed read behind
a condition whose row the staging does not hold: flagged, and 0, as in the
memory kernel."""

import numpy as np
import pytest

from tests import extra_model as X

pytestmark = pytest.mark.gpu

SPECIES = ["a", "b", "s", "g"]
# (the planning traces ssyn's condition with averages up to 7.25: what it reads
# above 20 is staged only as far as other reads ask for it)
REACTIONS = [
    ("asyn", True, "return c.getRate(asyn) / (1.0 + 0.01 * c.getCon(b, 5)) + 0.02 * c.getCon(a, c.getDelay(dreact_asyn));",
     {"a": 1}),
    ("adeg", False, "return c.getRate(adeg) * c.getCon(a);", {"a": -1}),
    ("bsyn", True, "return c.getRate(bsyn) * c.calculateNeighborAvg(s, 3) + 0.05 * c.calculateNeighborAvg(s) "
     "+ 0.01 * c.getCon(b, c.getDelay(dreact_bsyn));", {"b": 1}),
    ("bdeg", False, "return c.getRate(bdeg) * c.getCon(b);", {"b": -1}),
    ("ssyn", True, "double n = c.calculateNeighborAvg(s); if (n > 20.0) return c.getRate(ssyn) + "
     "0.2 * c.getCon(a, c.getDelay(dreact_ssyn)) + 0.1 * c.getCon(g, c.getDelay(dreact_asyn)); "
     "return 2.0 * c.getRate(ssyn) + "
     "0.01 * c.calculateNeighborAvg(g, c.getDelay(dreact_ssyn));", {"s": 1}),
    ("sdeg", False, "return c.getRate(sdeg) * c.getCon(s);", {"s": -1}),
    # delay 0 is the oldest row, 1 the newest
    ("gsyn", True, "return c.getRate(gsyn) + 0.01 * c.getCon(a, 0) + 0.02 * c.getCon(b, 1) + 0.01 * c.getCon(s, 2) "
     "+ 0.01 * c.getCon(g, c.getDelay(dreact_gsyn));", {"g": 1}),
    ("gdeg", False, "return c.getRate(gdeg) * c.getCon(g);", {"g": -1}),
]
MODEL = ("plain_reads", (SPECIES, [], REACTIONS))
RATES = [12.0, 0.4, 0.8, 0.5, 4.0, 0.4, 5.0, 0.3]


def _sets(cells, per_cell, delays, seed, count=2, duration=2.0, schedule=0):
    from dense_b200.engine import ParameterSet
    from dense_b200.tissue import default_graph
    rng = np.random.Generator(np.random.PCG64(seed))
    off, ids = default_graph(cells, 4)
    out = []
    for i in range(count):
        p = np.array(RATES + list(delays)) * np.concatenate([rng.uniform(0.7, 1.4, size=len(RATES)), np.ones(4)])
        cell = p[None, :] * np.concatenate([rng.uniform(0.8, 1.2, size=(cells, len(RATES))), np.ones((cells, 4))], 1)
        # s comes to 18-22 from below and from above
        ic = np.concatenate([rng.uniform(0.0, 30.0, size=2), [4.0 if i % 2 else 30.0], rng.uniform(0.0, 30.0, size=1)])
        out.append(ParameterSet(off, ids, p, cell_params=cell if per_cell else None, duration=duration,
                                schedule=schedule, init_conc=ic))
    return out


@pytest.mark.parametrize("per_cell", [False, True])
@pytest.mark.parametrize("cells", [1, 40, 200, 256, 300])
def test_plain_and_late_reads_match_the_oracle(cells, per_cell):
    sets = _sets(cells, per_cell, (7.0, 4.0, 6.0, 3.0), cells, count=4)
    want = X.oracle_states(X.oracle_library(*MODEL), sets, 0.01, 0.1)
    got, status = X.engine_states(X.engine_library(*MODEL), sets, 0.01, 0.1)
    assert (status == 0).all()
    for w, g in zip(want, got):
        assert np.array_equal(w, g)


@pytest.mark.parametrize("cells", [40, 300])
def test_late_flagged_reads(cells):
    """asyn's delay, with which ssyn reads g, reaches back further than the
    staged rows of g (eight)."""
    from dense_b200 import engine as E
    lib = X.engine_library(*MODEL)

    def run(schedule):
        return X.engine_states(lib, _sets(cells, False, (30.0, 4.0, 6.0, 3.0), 7, schedule=schedule), 0.01, 0.1)

    (got, flags), (want, want_flags) = run(E.SCHEDULE_REGISTER), run(E.SCHEDULE_MEMORY)
    assert (want_flags & 4).any()  # DENSE_SET_UNSTAGED_LAG
    assert np.array_equal(flags, want_flags)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


def test_late_flagged_reads_in_shared_rows():
    """The wave kernel keeps exactly the rows that the planning asked for; a
    read further back is flagged and stays within them."""
    from dense_b200 import engine as E
    lib = X.engine_library(*MODEL)
    for cells in (1, 40, 200):
        sets = _sets(cells, False, (30.0, 4.0, 6.0, 3.0), 7, schedule=E.SCHEDULE_SHARED_ROWS)
        states, flags = X.engine_states(lib, sets, 0.01, 0.1)
        assert (flags == 4).any() and all(np.isfinite(x).all() for x in states)
        sets = _sets(cells, False, (7.0, 4.0, 6.0, 3.0), 7, schedule=E.SCHEDULE_SHARED_ROWS)
        want = X.oracle_states(X.oracle_library(*MODEL), sets, 0.01, 0.1)
        states, flags = X.engine_states(lib, sets, 0.01, 0.1)
        assert (flags == 0).all() and all(np.array_equal(x, y) for x, y in zip(states, want))
