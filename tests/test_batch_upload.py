"""What a batch's creation copies to the device: small parts together, large
ones each from where they are (not through a second copy on the host)."""

import pytest

from tests.fake_cuda import calls

PROGRAM = """
from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from dense_b200 import engine as E
E.Batch(N.engine_library(N.NETWORK), _sets(%d, %r, 1, count=%d), 0.01, 0.1, [], precision=%d).close()
"""


@pytest.mark.parametrize("precision,width", [(0, 8), (1, 4)])
def test_large_parameters_are_copied_from_where_they_are(precision, width, tmp_path):
    params = 47  # of the network: reactions, delays, critical values
    log = calls(PROGRAM % (200, True, 60, precision), tmp_path)
    sizes = [int(x.split()[1]) for x in log if x.startswith("upload")]
    assert width * 200 * 60 * params in sizes
    assert sum(sizes) < width * 200 * 60 * params + (1 << 20)


def test_small_batches_are_one_copy(tmp_path):
    log = calls(PROGRAM % (200, False, 60, 0), tmp_path)
    assert sum(x.startswith("upload") for x in log) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("cells,count", [(200, 60), (300, 24), (200, 1100)])
def test_large_parts_match_the_oracle(cells, count):
    """Per-cell parameters above the staged size; and 1100 sets, whose
    descriptions are."""
    from tests import network_model as N
    from tests.test_step_reads_gpu import _sets
    sets = _sets(cells, count < 1000, 5, count=count, duration=0.3)
    picked = [0, count // 2, count - 1]
    got = N.engine_states(N.NETWORK, sets, 0.01, 0.1)
    N.assert_same(N.oracle_states(N.NETWORK, [sets[i] for i in picked], 0.01, 0.1), [got[i] for i in picked])
