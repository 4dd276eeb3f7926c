"""Device memory that a dropped batch leaves in the pool (host logic, with a
fake of the CUDA runtime): bounded, used by the next batch, and given back to
a batch that would not fit beside it."""

import pytest

from tests.fake_cuda import calls

MAKE = """
from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from dense_b200 import engine as E
lib = N.engine_library(N.NETWORK)
def batch(count):
    return E.Batch(lib, _sets(200, False, 1, count=1) * count, 0.01, 0.1, [])
"""
MB = 1 << 20


def _sizes(log, name):
    return [int(x.split()[1]) for x in log if x.startswith(name + " ") and x.endswith("ok")]


def test_a_batch_that_needs_what_the_pool_keeps(tmp_path):
    log = calls(MAKE + "batch(1500).close()\nbatch(3000).close()\n", tmp_path)
    small, large = _sizes(log, "pool_malloc")[0], _sizes(log, "malloc")[0]
    assert small < 512 * MB < large
    # a device that holds the larger batch, but not beside the smaller one
    capacity = large + small // 2
    log = calls(MAKE + "batch(1500).close()\nbatch(3000).close()\n", tmp_path, FAKE_CAPACITY=capacity)
    assert _sizes(log, "malloc") == [large]
    # and the pool serves again afterwards
    log = calls(MAKE + "batch(1500).close()\nbatch(3000).close()\nbatch(1500).close()\n", tmp_path,
                FAKE_CAPACITY=capacity)
    assert _sizes(log, "pool_malloc") == [small, small]


def test_a_batch_that_never_fits_is_refused(tmp_path):
    log = calls(MAKE + """
import pytest
with pytest.raises(E.DenseError, match="out of memory"):
    batch(3000)
batch(10).close()
""", tmp_path, FAKE_CAPACITY=100 * MB)
    assert len(_sizes(log, "pool_malloc")) == 1 and not _sizes(log, "malloc")


@pytest.mark.parametrize("count", [1, 1500])
def test_the_pool_keeps_at_most_half_a_gigabyte(count, tmp_path):
    log = calls(MAKE + "a = batch(%d)\nb = batch(%d)\na.close()\nb.close()\n" % (count, count), tmp_path)
    held = [int(x.split()[3]) for x in log if x.startswith("pool_free")]
    assert len(held) == 2 and held[-1] <= 512 * MB


def test_models_share_one_pool_per_device(tmp_path):
    """Each model is a library of its own; the memory that they keep together
    is bounded."""
    log = calls(MAKE + """
from tests.test_wave_gpu import _grid
grid = N.engine_library(N.GRID)
for device in (0, 1):
    E.Batch(lib, _sets(200, False, 1, count=1) * 20, 0.01, 0.1, [], device=device).close()
    E.Batch(grid, _grid(100, 10, 3, duration=2.0), 0.01, 0.1, [], device=device).close()
""", tmp_path)
    assert [x for x in log if x.startswith("pool dev")] == ["pool dev 0", "pool dev 1"]
    sizes, held = _sizes(log, "pool_malloc"), [int(x.split()[3]) for x in log if x.startswith("pool_free")]
    assert sizes[1] < sizes[0] and held[0] == held[1]  # the second model's batch is served from what the first left
