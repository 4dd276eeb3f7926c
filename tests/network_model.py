"""The gene-network and grid models of perf/cases.py for tests: their engine
libraries and their oracle, compiled from the same headers (no DENSE tree is
needed), and runs of both on the same sets."""

import importlib.util
import os

import numpy as np

from tests.conftest import ROOT

_spec = importlib.util.spec_from_file_location("perf_cases_models", os.path.join(ROOT, "perf", "cases.py"))
cases = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(cases)

NETWORK, GRID = cases.NETWORK, cases.GRID


def engine_library(model):
    return cases._library(model)


def oracle_library(model):
    from dense_b200 import models
    from oracle.pyoracle import load_oracle
    cases._library(model)
    before = os.environ.get(models.ENV)
    os.environ[models.ENV] = cases._tree[0]
    try:
        return load_oracle(model)
    finally:
        os.environ.pop(models.ENV) if before is None else os.environ.update({models.ENV: before})


def oracle_states(model, sets, dt, interval, analyses=()):
    """Final state of each set, and each set's oscillation / basic outputs,
    from the oracle.  sets: ParameterSets; analyses: engine Analysis objects
    (Basic and Oscillation)."""
    from dense_b200 import engine as E
    O = oracle_library(model)
    out = []
    for s in sets:
        cell = s.cell_params if s.cell_params is not None else np.tile(s.set_params, (s.num_cells, 1))
        sim = O.create(s.nbr_offsets, s.nbr_ids, cell, s.set_params, s.init_conc, dt, s.perturb)
        for a in analyses:
            if a.kind == E.BASIC:
                sim.add_basic(a.species, a.cell_start, a.cell_end, a.time_start, a.time_end)
            else:
                sim.add_oscillation(a.species, a.cell_start, a.cell_end, a.time_start, a.time_end, a.win_range,
                                    a.anlys_intvl)
        sim.run(s.duration, interval)
        r = {"state": sim.state()}
        for k, a in enumerate(analyses):
            r[k] = sim.basic(k) if a.kind == E.BASIC else sim.oscillation(k)
        out.append(r)
    return out


def engine_states(model, sets, dt, interval, analyses=(), precision=0, chunks=None, graph=False):
    """The same from the engine, with each set's status; `chunks` splits the
    run into launches of so many chunks."""
    from dense_b200 import engine as E
    b = E.Batch(engine_library(model), sets, dt, interval, list(analyses), precision=precision)
    if chunks is None:
        b.run(graph=graph)
    else:
        total = max(int(np.ceil(s.duration / interval)) for s in sets)
        for _ in range(0, total, chunks):
            b.run(chunks, graph=graph)
    b.sync()
    status = b.status()
    out = []
    for i in range(len(sets)):
        r = {"state": b.state(i), "status": int(status[i])}
        for k, a in enumerate(analyses):
            if a.kind in (E.BASIC, E.OSCILLATION):
                r[k] = b.basic(k, i) if a.kind == E.BASIC else b.oscillation(k, i)
        out.append(r)
    b.close()
    return out


def assert_same(want, got):
    """Bit equality (every NaN equal to every NaN) of two results' arrays."""
    for i, (w, g) in enumerate(zip(want, got)):
        for key, v in w.items():
            for name, x in (v.items() if isinstance(v, dict) else [("", v)]):
                y = g[key][name] if name else g[key]
                assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=np.asarray(x).dtype.kind == "f"), \
                    (i, key, name)
