"""dense_engine_plan_ctas: how many CTAs a set is spread over, by cells, hints
and analyses, as dense_engine_create then launches them."""

import numpy as np
import pytest

from dense_b200 import engine as E
from tests import network_model as N
from tests.fake_cuda import calls
from tests.test_step_reads_gpu import _sets


def _ctas(cells, analyses=(), **hint):
    lib = N.engine_library(N.NETWORK)
    return E.plan_ctas(lib, [_sets(cells, False, 1, count=1, **hint)[0]], 0.01, 0.1, analyses)[0]


@pytest.mark.parametrize("cells,want", [(1, 1), (256, 1), (257, 2), (512, 2), (513, 3), (4096, 16), (4097, 1)])
def test_by_cells(cells, want, tmp_path):
    assert _ctas(cells) == want
    log = calls("""
from tests import network_model as N
from tests.test_step_reads_gpu import _sets
from dense_b200 import engine as E
b = E.Batch(N.engine_library(N.NETWORK), _sets(%d, False, 1, count=1), 0.01, 0.1, [])
b.run()
""" % cells, tmp_path)
    launched = [int(x.split()[1]) for x in log if x.startswith("cluster_launch")]
    assert launched == ([want] if want > 1 else [])


def test_hints_keep_one_cta():
    assert _ctas(700, schedule=E.SCHEDULE_MEMORY) == 1
    s = _sets(700, False, 1, count=1)[0]
    s.mem_block = 128
    lib = N.engine_library(N.NETWORK)
    assert E.plan_ctas(lib, [s], 0.01, 0.1)[0] == 1
    _, kernel, _ = E.plan(lib, [s], 0.01, 0.1)
    assert kernel[0] == 128
    assert _ctas(700, [E.Analysis.basic(list(range(14)), 0, 700)]) == 3


def test_null_arguments():
    import ctypes as C
    f = N.engine_library(N.NETWORK).lib.dense_engine_plan_ctas
    f.argtypes = None
    assert f(None, 0, None, None) != 0
    assert f(None, C.c_int(1), None, np.zeros(1, np.int32).ctypes.data_as(C.c_void_p)) != 0
