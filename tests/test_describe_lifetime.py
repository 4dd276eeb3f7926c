"""Arrays that a set makes each time it is asked for them live as long as the
descriptors that hold their addresses."""

import ctypes as C
import gc

import numpy as np

from dense_b200 import engine as E
from dense_b200.tissue import default_graph
from tests.test_batch_setup import _Model


class MadeOnAccess(E.ParameterSet):
    @property
    def set_params(self):
        return self._p * 1.0

    @set_params.setter
    def set_params(self, v):
        self._p = v

    @property
    def nbr_ids(self):
        return self._ids.copy()

    @nbr_ids.setter
    def nbr_ids(self, v):
        self._ids = v


def test_descriptors_hold_arrays_made_on_access():
    rng = np.random.Generator(np.random.PCG64(1))
    off, ids = default_graph(12, 4)
    params = [rng.uniform(size=7) for _ in range(50)]
    run, cset, keep = E._describe(_Model, [MadeOnAccess(off, ids, p, duration=1.0) for p in params], [], 0.01, 0.1,
                                  E.FP64, 0)
    gc.collect()
    scribble = [np.full(7, -1.0) for _ in range(200)] + [np.full(len(ids), -1, np.int32) for _ in range(200)]
    places = set()
    for c, p in zip(cset, params):
        assert list(c.set_params[:7]) == list(p)
        assert list(c.nbr_ids[:len(ids)]) == list(ids)
        places.add(C.cast(c.set_params, C.c_void_p).value)
    assert len(places) == 50 and len(scribble) == 400 and keep and run is not None
