"""The whole-network entry points: every declared symbol is exported, and
bad arguments are refused before any CUDA call (so this runs without a GPU)."""

import ctypes as C
import os
import re

from tests.conftest import ROOT


def test_declared_symbols_are_exported():
    from dense_b200 import surrogate
    lib = C.CDLL(surrogate.build())
    text = open(os.path.join(ROOT, "include", "dense_b200_network.h")).read()
    names = set(re.findall(r"^int(?:64_t)? (dense_mlp_[a-z0-9_]+)\(", text, re.M))
    assert len(names) == 8, names
    for name in names:
        assert hasattr(lib, name), name


def test_bad_arguments_are_refused():
    from dense_b200 import surrogate
    L = surrogate.lib()
    p = C.c_void_p(4096)  # never dereferenced: every call below is refused first
    four = (C.c_void_p * 4)(4096, 4096, 4096, 4096)
    odd = (C.c_void_p * 4)(4096, 4100, 4096, 4096)
    none = (C.c_void_p * 4)()
    assert L.dense_mlp_pack(none, p, 1, None) == 1
    assert L.dense_mlp_pack(four, C.c_void_p(4104), 1, None) == 1
    for rows, n_in, ldx, n_out, bias in ((-1, 44, 44, 5, four), (8, 65, 65, 5, four), (8, 0, 1, 5, four),
                                         (8, 44, 43, 5, four), (8, 44, 44, 129, four), (8, 44, 44, 0, four),
                                         (8, 44, 44, 5, odd)):
        assert L.dense_mlp_predict(p, ldx, rows, n_in, p, bias, n_out, p, p, None) == 1
    assert L.dense_mlp_predict(None, 44, 0, 44, p, four, 5, None, p, None) == 0  # nothing to do
    m = (C.c_float * 8)()
    rank = lambda nets, n_out, tol, spread: L.dense_mlp_rank(  # noqa: E731
        p, 45, 8, p, p, 44, spread, nets, four, four, n_out, m, m, 0.1, 30.0, tol, 50.0, 0.1, p, p, None)
    assert rank(0, 5, 3.0, 1.4) == rank(65, 5, 3.0, 1.4) == rank(1, 4, 3.0, 1.4) == rank(1, 9, 3.0, 1.4) == 1
    assert rank(1, 5, 0.0, 1.4) == rank(1, 5, 3.0, 0.0) == 1
    need = L.dense_mlp_train_bytes(300, 5)
    assert need > 0 and L.dense_mlp_train_bytes(0, 5) == L.dense_mlp_train_bytes(300, 129) == 0
    assert L.dense_mlp_train_pass(p, 44, 300, 44, p, p, 5, None, 300, p, four, None, 1.0, p, p, need - 1, p, None) == 1
    assert L.dense_mlp_train_pass(p, 44, 300, 44, p, p, 5, None, 0, p, four, None, 1.0, p, p, need, p, None) == 1
    none6 = [None] * 6
    assert L.dense_mlp_train_finish(p, need, 300, 5, None, None, None, *none6, None, None) == 1  # nothing asked for
    assert L.dense_mlp_train_finish(p, need, 300, 5, None, None, p, *none6, p, None) == 1       # Adam without weights
    assert L.dense_mlp_train_finish(p, need - 1, 300, 5, four, four, None, *none6, None, None) == 1
    epoch = lambda steps, idx, hyper: L.dense_mlp_train_epoch(  # noqa: E731
        p, 44, 300, 44, p, p, 5, idx, 300, steps, hyper, p, p, need - 1, *[four] * 6, p, p, None)
    assert epoch(1, p, p) == epoch(-1, p, p) == epoch(0, None, p) == epoch(0, p, None) == 1
    assert epoch(0, p, p) == 0
