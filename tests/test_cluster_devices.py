"""Where sets of 257 to 4096 cells run (host logic, with a fake of the CUDA
runtime in place of a GPU): over clusters on every device that a process uses,
in the memory kernel where the device holds no cluster of that size."""

import pytest

from tests.fake_cuda import calls

PROGRAM = """
from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from dense_b200 import engine as E
for device in %r:
    b = E.Batch(N.engine_library(N.NETWORK), _sets(%d, False, 1, count=2), 0.01, 0.1, [], precision=%d, device=device)
    b.run()
    b.sync()
    b.close()
"""


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("cells", [300, 4000])
def test_every_device_is_opted_in(cells, precision, tmp_path):
    log = calls(PROGRAM % ((0, 1, 0), cells, precision), tmp_path)
    for dev in (0, 1):
        mine = [x for x in log if x.endswith("dev %d" % dev)]
        first = next(i for i, x in enumerate(mine) if x.startswith("cluster_launch"))
        assert any(x.startswith("attribute 8 100000") for x in mine[:first])   # dynamic shared memory
        assert any(x.startswith("attribute 14 1") for x in mine[:first])       # clusters of more than eight
    ranks = (cells + 255) // 256
    assert sum(x.startswith("cluster_launch %d x" % (2 * ranks)) for x in log) == 3


@pytest.mark.parametrize("precision", [0, 1])
def test_memory_kernel_where_no_cluster_fits(precision, tmp_path):
    log = calls(PROGRAM % ((0,), 3000, precision), tmp_path, FAKE_CLUSTERS=0)
    assert not any(x.startswith("cluster_launch") for x in log)
    assert any(x.startswith("launch 2 x 256") for x in log)
