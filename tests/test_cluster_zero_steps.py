"""A concentration check over a cluster when no step lies between two samples
(an interval below the step size): the CTAs read each other's flags after a
sample, so a cluster barrier has to come between those reads and the next
sample that may set one (from the source), and the set is dropped at the same
sample as in the memory kernel."""

import re

import numpy as np
import pytest

from tests import network_model as N
from tests.test_cluster_counters import _register_kernel
from tests.test_step_reads_gpu import _sets


def test_a_chunk_opens_with_a_cluster_barrier_when_flags_may_be_read_still():
    body = _register_kernel()
    opening = body[body.index("const int row = a.val_slot[sp];"):body.index("analyses_sample<")]
    assert re.search(r"if \(kCluster && \(folds \|\| \(checks && steps_per_chunk == 0\)\)\) \{\s*cluster_barrier\(\);",
                     opening)


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [40.0, 60.0])
def test_dropped_at_the_same_sample_as_in_the_memory_kernel(limit):
    from dense_b200 import engine as E
    cells = 700
    # checked from 0.0045 on, i.e. the tenth sample; the states stand still
    an = [E.Analysis.conccheck([0], 0, cells, -1.0, limit, 0.0045)]

    def run(schedule):
        sets = _sets(cells, False, 4, count=60, duration=0.02, schedule=schedule)
        for s in sets:
            s.init_conc[0] = 50.0
        b = E.Batch(N.engine_library(N.NETWORK), sets, 0.01, 0.0005, an)
        b.run()
        b.sync()
        out = b.status(), b.progress()[0], np.stack([b.state(i) for i in (0, 30, 59)])
        b.close()
        return out

    got, want = run(E.SCHEDULE_AUTO), run(E.SCHEDULE_MEMORY)
    assert bool(got[0][0] & E.SET_DROPPED) == (limit < 50.0)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
