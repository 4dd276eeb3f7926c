"""Step loads issued before the barrier that ends the step before, and behind
it where a neighbour's row of the step itself is read: delays from zero to a
few steps, one parameter row or one per cell (so that only some cells read
the newest row), in one CTA and over a cluster, in chunks of one step and of
several, against the oracle bit for bit; FP32 against the memory kernel."""

import numpy as np
import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("delays", [[0.0], [0.01], [0.0, 0.01], [0.01, 0.02], [0.02, 0.03, 0.05]])
@pytest.mark.parametrize("cells,per_cell", [(1, False), (40, False), (90, True), (256, False), (300, False), (300, True)])
def test_shortest_delays(cells, per_cell, delays):
    sets = _sets(cells, per_cell, cells, count=3, delays=delays, duration=0.5)
    N.assert_same(N.oracle_states(N.NETWORK, sets, 0.01, 0.05), N.engine_states(N.NETWORK, sets, 0.01, 0.05, chunks=3))


@pytest.mark.parametrize("interval", [0.01, 0.03])
@pytest.mark.parametrize("cells", [64, 300])
def test_chunks_of_few_steps(cells, interval):
    from dense_b200.engine import Analysis
    an = [Analysis.basic([0, 13], 0, cells)]
    sets = _sets(cells, False, 2, count=160 if cells == 64 else 2, delays=[0.01, 0.05], duration=0.3)
    got = N.engine_states(N.NETWORK, sets, 0.01, interval, an)
    N.assert_same(N.oracle_states(N.NETWORK, sets[:3], 0.01, interval, an), got[:3])


@pytest.mark.parametrize("cells", [70, 300])
def test_fp32(cells):
    from dense_b200 import engine as E
    run = lambda schedule: N.engine_states(  # noqa: E731
        N.NETWORK, _sets(cells, False, 7, delays=[0.0, 0.01, 0.04], duration=0.5, schedule=schedule), 0.01, 0.05,
        precision=E.FP32_KAHAN)
    for g, w in zip(run(E.SCHEDULE_AUTO), run(E.SCHEDULE_MEMORY)):
        assert g["status"] == w["status"] and np.array_equal(g["state"], w["state"], equal_nan=True)
