"""Batch set-up: the set descriptors handed to the C ABI, tissues that
several sets share, and batches made and dropped while others run."""

import ctypes as C
import threading

import numpy as np
import pytest

from dense_b200 import engine as E
from dense_b200.tissue import default_graph


class _Model:  # what _describe reads of a model library
    num_params = 7

    @staticmethod
    def species_ids(names):
        return list(names)


def test_descriptors_hold_every_field_of_every_set():
    rng = np.random.Generator(np.random.PCG64(1))
    off, ids = default_graph(12, 4)
    sets = [E.ParameterSet(off, ids, rng.uniform(size=7),
                           cell_params=rng.uniform(size=(12, 7)) if i % 2 else None,
                           init_conc=rng.uniform(size=3) if i % 3 else None,
                           perturb=rng.uniform(size=4) if i == 2 else None,
                           duration=1.5 * i, schedule=i % 7, mem_block=32 * (i % 3)) for i in range(6)]
    _, cset, _ = E._describe(_Model, sets, [], 0.01, 0.1, E.FP64, 0)
    assert len(cset) == 6
    for s, c in zip(sets, cset):
        assert (c.num_cells, c.duration, c.schedule, c.mem_block) == (12, s.duration, s.schedule, s.mem_block)
        for name in ("nbr_offsets", "nbr_ids", "set_params", "cell_params", "init_conc", "perturb"):
            a, p = getattr(s, name), getattr(c, name)
            assert (C.cast(p, C.c_void_p).value or 0) == (0 if a is None else a.ctypes.data), name


def test_wrong_parameter_counts_are_refused():
    off, ids = default_graph(4, 2)
    with pytest.raises(E.DenseError, match="set_params"):
        E._describe(_Model, [E.ParameterSet(off, ids, np.zeros(6))], [], 0.01, 0.1, E.FP64, 0)
    with pytest.raises(E.DenseError, match="cell_params"):
        E._describe(_Model, [E.ParameterSet(off, ids, np.zeros(7), cell_params=np.zeros((3, 7)))], [], 0.01, 0.1,
                    E.FP64, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(40, 40, 40), (40, 300, 40), (300, 300, 12)])
def test_shared_tissues_equal_copied_ones(cells):
    from tests import network_model as N
    from tests.test_step_reads_gpu import _sets
    shared = [_sets(n, False, 20 + k, count=1)[0] for k, n in enumerate(cells)]
    first = {}
    for s in shared:  # sets of one size share the arrays of the first
        f = first.setdefault(s.num_cells, s)
        s.nbr_offsets, s.nbr_ids = f.nbr_offsets, f.nbr_ids
    want = N.engine_states(N.NETWORK, [_sets(n, False, 20 + k, count=1)[0] for k, n in enumerate(cells)], 0.01, 0.1)
    N.assert_same(want, N.engine_states(N.NETWORK, shared, 0.01, 0.1))


@pytest.mark.gpu
def test_batches_made_and_dropped_in_two_threads():
    from tests import network_model as N
    from tests.test_step_reads_gpu import _sets
    sizes = [(10, 3), (200, 60), (64, 1), (300, 5)]
    want = [N.engine_states(N.NETWORK, _sets(c, False, 30 + c, count=k), 0.01, 0.1) for c, k in sizes]
    bad = []

    def work(order):
        try:
            for _ in range(4):
                for i in order:
                    c, k = sizes[i]
                    N.assert_same(want[i], N.engine_states(N.NETWORK, _sets(c, False, 30 + c, count=k), 0.01, 0.1))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=(o,)) for o in ([0, 1, 2, 3], [3, 1, 0, 2])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
