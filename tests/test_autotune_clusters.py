"""The tuner times the cluster kernel for the sets the engine would run in it,
and does not take over choices cached before that kernel was one of them."""

import json

import pytest

from dense_b200 import engine as E
from dense_b200.autotune import Autotuner, candidates, schedules
from tests import network_model as N
from tests.test_step_reads_gpu import _sets


@pytest.mark.parametrize("log2", range(1, 17))
def test_schedules_of_a_bucket(log2):
    got = schedules(False, log2)
    assert ((E.SCHEDULE_AUTO, 0) in got) == (log2 <= 12)
    assert [c for c in got if c[0] != E.SCHEDULE_AUTO] == [c for c in candidates(False, log2) if c[0] != E.SCHEDULE_AUTO]
    assert len(set(got)) == len(got)
    assert schedules(True, log2) == candidates(True, log2)


def test_cluster_sets_are_tuned_with_the_cluster_kernel(tmp_path):
    cache = tmp_path / "tune.json"
    # a choice from before the cluster kernel
    cache.write_text(json.dumps({"fake|signal_network|0|10": [E.SCHEDULE_MEMORY, 256]}))
    timed = []

    def timer(model, sample, schedule, mem_block, step_size, minutes, device=0):
        timed.append((schedule, mem_block))
        return 2.0 if schedule == E.SCHEDULE_AUTO else 1.0

    lib = N.engine_library(N.NETWORK)
    sets = [_sets(n, False, n, count=1)[0] for n in (600, 900, 1000)]
    chosen = Autotuner(cache_path=str(cache), timer=timer, gpu_name="fake").tune(N.NETWORK, sets, 0.01)
    assert lib is not None and (E.SCHEDULE_AUTO, 0) in timed and (E.SCHEDULE_MEMORY, 256) in timed
    assert chosen == {(False, 10): (E.SCHEDULE_AUTO, 0)}
    assert all((s.schedule, s.mem_block) == (E.SCHEDULE_AUTO, 0) for s in sets)
    timed.clear()
    again = [_sets(900, False, 1, count=1)[0]]
    assert Autotuner(cache_path=str(cache), timer=timer, gpu_name="fake").tune(N.NETWORK, again, 0.01) == chosen
    assert timed == []
