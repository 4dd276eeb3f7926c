"""Further models for tests, in the form of perf/cases.py's: headers written to
a folder of their own, the engine library and the oracle compiled from them."""

import os
import tempfile

from tests import network_model as N

_trees = {}


def _with_tree(name, definition, make):
    """make() with the model's folder named by the environment."""
    from dense_b200 import models
    if name not in _trees:
        _trees[name] = tempfile.mkdtemp(prefix="dense_%s_" % name)
        folder = os.path.join(_trees[name], "models", name)
        os.makedirs(folder)
        for f, lines in N.cases._headers(*definition).items():
            path = os.path.join(folder, f)
            with open(path, "w") as h:
                h.write("\n".join(lines) + "\n")
            os.utime(path, (0, 0))  # a library built before is not older than its model
        models.MODEL_DIRS[name] = "models/" + name
    before = os.environ.get(models.ENV)
    os.environ[models.ENV] = _trees[name]
    try:
        return make()
    finally:
        models.MODEL_DIRS.pop(name)
        del _trees[name]
        os.environ.pop(models.ENV) if before is None else os.environ.update({models.ENV: before})


def engine_library(name, definition):
    from dense_b200 import build
    from dense_b200.engine import ModelLibrary
    return ModelLibrary(_with_tree(name, definition, lambda: build.build_model(name)))


def oracle_library(name, definition):
    from oracle.pyoracle import load_oracle
    return _with_tree(name, definition, lambda: load_oracle(name))


def oracle_states(lib, sets, dt, interval):
    """Final state of each set from an oracle library."""
    import numpy as np
    out = []
    for s in sets:
        cell = s.cell_params if s.cell_params is not None else np.tile(s.set_params, (s.num_cells, 1))
        sim = lib.create(s.nbr_offsets, s.nbr_ids, cell, s.set_params, s.init_conc, dt, s.perturb)
        sim.run(s.duration, interval)
        out.append(sim.state())
    return out


def engine_states(lib, sets, dt, interval, precision=0):
    """(states, statuses) of an engine library's batch."""
    from dense_b200 import engine as E
    b = E.Batch(lib, sets, dt, interval, [], precision=precision)
    b.run()
    b.sync()
    out = [b.state(i) for i in range(len(sets))], b.status()
    b.close()
    return out
