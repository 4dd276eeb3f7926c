"""The sample counters of a set spread over a cluster: each CTA copies them
when a launch begins and rank 0 writes their successors at the first sample,
so the copies come before that in every CTA (read from the source: a CTA that
starts late is a matter of the GPU's scheduling).  And chunked launches of
many clusters, whose CTAs do start at their own times, against the oracle."""

import os
import re

import numpy as np
import pytest

from tests import network_model as N
from tests.conftest import ROOT
from tests.test_step_reads_gpu import _sets


def _register_kernel():
    with open(os.path.join(ROOT, "dense_b200", "csrc", "engine", "step_kernel.cuh")) as f:
        src = f.read()
    start = src.index("dense_step_kernel(const StepArgs a")
    return src[start:src.index("\n}\n", start)]


def test_counters_are_copied_before_a_cluster_barrier():
    body = _register_kernel()
    copied = body.index("s_samples[c] = anl[")
    sampled = body.index("analyses_sample<")
    between = body[copied:sampled]
    # one that every launch with analyses meets, ahead of the chunk loop
    assert re.search(r"if \(kCluster && a\.n_analyses > 0\) \{[^}]*cluster_barrier\(\);", between)


@pytest.mark.gpu
@pytest.mark.parametrize("chunks", [1, 3])
def test_chunked_launches_of_many_clusters(chunks):
    """Clusters of three CTAs, more than the GPU holds at once, recording
    trajectories and oscillations without a Basic analysis."""
    from dense_b200 import engine as E
    cells, count = 600, 150
    an = [E.Analysis.oscillation([0, 5], 0, cells, 0.0, float("inf"), 0.4, 0.1),
          E.Analysis.trajectory([0], 0, cells, 0.0, 1.0)]
    sets = _sets(cells, False, 11, count=count, duration=1.0)
    b = E.Batch(N.engine_library(N.NETWORK), sets, 0.01, 0.1, an)
    for _ in range(0, 10, chunks):
        b.run(chunks)
    b.sync()
    picked = [0, 50, 98, 99, 100, 149]
    got = [{"state": b.state(i), 0: b.oscillation(0, i)} for i in picked]
    recorded = [b.trajectory(1, i) for i in picked]
    b.close()
    N.assert_same(N.oracle_states(N.NETWORK, [sets[i] for i in picked], 0.01, 0.1, an[:1]), got)
    for times, values in recorded:
        assert values.shape == (10, 1, cells) and np.allclose(times, 0.1 * np.arange(10))
