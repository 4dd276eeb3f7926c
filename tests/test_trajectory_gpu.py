"""Recorded trajectories of sets of several warps: every sample is the state
the set had at that chunk, in every kernel that records one."""

import numpy as np
import pytest

from tests import network_model as N
from tests.test_step_reads_gpu import _sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [70, 200, 300])
def test_every_sample_is_recorded_once(cells):
    from dense_b200 import engine as E
    an = [E.Analysis.trajectory([0, 9], 0, cells, 0.0, 2.0)]
    sets = _sets(cells, False, cells, count=200)
    b = E.Batch(N.engine_library(N.NETWORK), sets, 0.01, 0.1, an)
    b.run()
    b.sync()
    picked = [0, 99, 199]
    got = {i: b.trajectory(0, i) for i in picked}
    b.reset()
    states = {i: [] for i in picked}
    for _ in range(20):
        for i in picked:
            states[i].append(b.state(i)[[0, 9]])
        b.run(1)
        b.sync()
    b.close()
    for i in picked:
        times, values = got[i]
        assert values.shape == (20, 2, cells)
        assert np.allclose(times, 0.1 * np.arange(20))
        # the first state is read before any launch wrote the state block back
        assert np.array_equal(values, np.stack(states[i])), i
