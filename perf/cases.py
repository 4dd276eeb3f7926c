"""The work this framework is timed on: sizes, inputs and calls.

Two families of cases:

* the simulation engine (``dense_b200.engine``), on two models in the
  framework's model-header form that this file writes out and compiles
  through ``dense_b200.build`` -- a delayed gene network with cell-to-cell
  signalling (the size of a segmentation-clock model: 14 species, 32
  reactions, 10 delays) and a two-species reaction-diffusion grid whose
  neighbour averages read the row being written (cell-ordered sets);
* the surrogate-screened search (``dense_b200.surrogate``,
  ``dense_b200.search``): training, gradients, prediction, ranking and the
  synchrony feature.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare`` makes inputs and what a program keeps, ``run`` is one
pass through the public entry points, ``work`` what the pass cannot do
without, and ``exact`` the same results in plain float64 torch.
"""

import os
import tempfile

import numpy as np
import torch

from dense_b200 import build as engine_build
from dense_b200 import engine as E
from dense_b200 import models, search, surrogate, workloads
from dense_b200.tissue import default_graph

DT = 0.01        # minutes per Euler step
INTERVAL = 0.1   # minutes between analysis samples (10 steps)

# ------------------------------------------------------------------ models

GENES = 4
NETWORK = "signal_network"
GRID = "diffusive_grid"

NETWORK_SPECIES = (["m%d" % g for g in range(GENES)] + ["p%d" % g for g in range(GENES)] +
                   ["d%d" % g for g in range(GENES)] + ["ms", "ps"])
NETWORK_CRITICAL = ["d%d" % g for g in range(GENES)] + ["ps"]
REPRESSOR = [2, 0, 1, 1]  # a ring of three genes and a fourth beside it


def _network_reactions():
    """(name, delayed, rate expression, {species: delta}) in list order."""
    out = []
    for g in range(GENES):
        up = REPRESSOR[g]
        # synthesis repressed by another gene's dimer (a second-order
        # Hill term, delayed); the first two genes are activated by the
        # neighbours' signal protein
        squared = ("double x = c.getCon(d{u}, c.getDelay(dreact_msyn{g})) / c.getCritVal(rcrit_d{u});"
                   .format(u=up, g=g))
        if g < 2:
            rate = (squared + " double s = c.calculateNeighborAvg(ps, c.getDelay(dreact_msyn{g})) / "
                    "c.getCritVal(rcrit_ps); return c.getRate(msyn{g}) * (1.0 + s) / (1.0 + s + x * x);".format(g=g))
        else:
            rate = squared + " return c.getRate(msyn{g}) / (1.0 + x * x);".format(g=g)
        out.append(("msyn%d" % g, True, rate, {"m%d" % g: 1}))
        out.append(("mdeg%d" % g, False, "return c.getRate(mdeg{g}) * c.getCon(m{g});".format(g=g), {"m%d" % g: -1}))
        out.append(("psyn%d" % g, True,
                    "return c.getRate(psyn{g}) * c.getCon(m{g}, c.getDelay(dreact_psyn{g}));".format(g=g),
                    {"p%d" % g: 1}))
        out.append(("pdeg%d" % g, False, "return c.getRate(pdeg{g}) * c.getCon(p{g});".format(g=g), {"p%d" % g: -1}))
        out.append(("bind%d" % g, False, "return c.getRate(bind{g}) * c.getCon(p{g}) * c.getCon(p{g});".format(g=g),
                    {"p%d" % g: -2, "d%d" % g: 1}))
        out.append(("dis%d" % g, False, "return c.getRate(dis{g}) * c.getCon(d{g});".format(g=g),
                    {"p%d" % g: 2, "d%d" % g: -1}))
        out.append(("ddeg%d" % g, False, "return c.getRate(ddeg{g}) * c.getCon(d{g});".format(g=g), {"d%d" % g: -1}))
    out.append(("mssyn", True, "double x = c.getCon(d0, c.getDelay(dreact_mssyn)) / c.getCritVal(rcrit_d0); "
                "return c.getRate(mssyn) / (1.0 + x * x);", {"ms": 1}))
    out.append(("msdeg", False, "return c.getRate(msdeg) * c.getCon(ms);", {"ms": -1}))
    out.append(("pssyn", True, "return c.getRate(pssyn) * c.getCon(ms, c.getDelay(dreact_pssyn));", {"ps": 1}))
    out.append(("psdeg", False, "return c.getRate(psdeg) * c.getCon(ps);", {"ps": -1}))
    return out


NETWORK_REACTIONS = _network_reactions()
NETWORK_DELAYED = [r[0] for r in NETWORK_REACTIONS if r[1]]

# the Brusselator with diffusion by neighbour averages of the row of one step
# back, which the cell-ordered update partly overwrites
GRID_SPECIES = ["u", "v"]
GRID_REACTIONS = [
    ("feed", False, "return c.getRate(feed);", {"u": 1}),
    ("conv", False, "return c.getRate(conv) * c.getCon(u);", {"u": -1, "v": 1}),
    ("turn", False, "return c.getRate(turn) * c.getCon(u) * c.getCon(u) * c.getCon(v);", {"u": 1, "v": -1}),
    ("loss", False, "return c.getRate(loss) * c.getCon(u);", {"u": -1}),
    ("diffu", False, "return c.getRate(diffu) * (c.calculateNeighborAvg(u, 1) - c.getCon(u));", {"u": 1}),
    ("diffv", False, "return c.getRate(diffv) * (c.calculateNeighborAvg(v, 1) - c.getCon(v));", {"v": 1}),
]


def _headers(species, critical, reactions):
    """The four model headers."""
    lists = ["#ifndef DELAY_REACTION", "#define DELAY_REACTION(name) REACTION(name)", "#define PLAIN_DELAYS", "#endif"]
    lists += ["%s(%s)" % ("DELAY_REACTION" if d else "REACTION", n) for n, d, _, _ in reactions]
    lists += ["#ifdef PLAIN_DELAYS", "#undef PLAIN_DELAYS", "#undef DELAY_REACTION", "#endif"]
    deltas, rates = ["#pragma once", '#include "core/reaction.hpp"'], ["#pragma once", '#include "core/reaction.hpp"']
    for n, _, rate, delta in reactions:
        deltas.append("STATIC_VAR int num_deltas_%s = %d;" % (n, len(delta)))
        deltas.append("STATIC_VAR int deltas_%s[] = {%s};" % (n, ", ".join(str(v) for v in delta.values())))
        deltas.append("STATIC_VAR specie_id delta_ids_%s[] = {%s};" % (n, ", ".join(delta)))
        rates.append("template <> template <class Ctxt> RATETYPE reaction<%s>::active_rate(const Ctxt& c) { %s }"
                     % (n, rate.replace("double ", "RATETYPE ")))
    return {"specie_list.hpp": ["%s(%s)" % ("CRITICAL_SPECIE" if s in critical else "SPECIE", s) for s in species],
            "reactions_list.hpp": lists, "reaction_deltas.hpp": deltas, "model_impl.hpp": rates}


MODELS = {NETWORK: (NETWORK_SPECIES, NETWORK_CRITICAL, NETWORK_REACTIONS), GRID: (GRID_SPECIES, [], GRID_REACTIONS)}
_tree = []


def _library(key):
    """The engine library of one of this file's models, compiled on first
    use (a program's own model joins MODEL_DIRS and its tree is named by the
    environment)."""
    if not _tree:
        _tree.append(tempfile.mkdtemp(prefix="dense_models_"))
        for name, (species, critical, reactions) in MODELS.items():
            folder = os.path.join(_tree[0], "models", name)
            os.makedirs(folder)
            for f, lines in _headers(species, critical, reactions).items():
                path = os.path.join(folder, f)
                with open(path, "w") as h:
                    h.write("\n".join(lines) + "\n")
                os.utime(path, (0, 0))  # a library built before is not older than its model
            models.MODEL_DIRS[name] = "models/" + name
        # a read-only installation keeps what it compiles elsewhere
        folder = engine_build.LIB_DIR if os.path.isdir(engine_build.LIB_DIR) else engine_build.HERE
        if not os.access(folder, os.W_OK) and not os.path.exists(engine_build.lib_path(key)):
            engine_build.LIB_DIR = os.path.join(tempfile.gettempdir(), "dense_b200_lib_%d" % os.getuid())
            engine_build.OBJ_DIR = os.path.join(engine_build.LIB_DIR, "obj")
    before = os.environ.get(models.ENV)
    os.environ[models.ENV] = _tree[0]
    try:
        return E.load(key)
    finally:
        os.environ.pop(models.ENV) if before is None else os.environ.update({models.ENV: before})


def _network_template():
    """Parameters of the network, [rates | delays | critical values]."""
    value = {"msyn": 33.0, "mdeg": 0.3, "psyn": 4.5, "pdeg": 0.35, "bind": 0.02, "dis": 0.1, "ddeg": 0.35}
    rates = []
    for n, _, _, _ in NETWORK_REACTIONS:
        rates.append({"mssyn": 25.0, "msdeg": 0.28, "pssyn": 2.0, "psdeg": 0.3}.get(n) or value[n.rstrip("0123456789")])
    delays = [8.0 + 1.1 * i if n[0] == "m" else 3.0 + 0.4 * i for i, n in enumerate(NETWORK_DELAYED)]
    return np.array(rates + delays + [240.0, 230.0, 250.0, 220.0, 420.0])


GRID_TEMPLATE = np.array([1.0, 2.6, 1.0, 1.0, 0.8, 0.25])

# ------------------------------------------------------------------- cases

MARKER = NETWORK_SPECIES.index("m0")


def listed():
    def engine(name, **kw):
        d = {"name": name, "path": "engine", "model": NETWORK, "sets": 1, "cells": 200, "width": 4, "minutes": 10.0,
             "bits": 64, "analyses": "oscillation", "cell_params": False, "kept": False}
        return dict(d, **kw)

    return [
        # the smallest call: a regression-test tissue, one analysis
        engine("ten_cells", cells=10, width=5, minutes=1.0, analyses="basic"),
        # one tissue with every parameter of every cell perturbed, all
        # analyses: the usual single simulation
        engine("one_tissue", minutes=10.0, analyses="all", cell_params=True),
        # one generation of a parameter search: new sets simulated, their
        # oscillation features read back
        engine("search_generation", sets=1024, minutes=5.0),
        # the large batch, kept on the GPU and run again from its start
        engine("batch_fp64", sets=4096, minutes=3.0, kept=True),
        # the same in the FP32 mode with compensated state
        engine("batch_fp32", sets=2000, minutes=3.0, bits=32, kept=True),
        # tissues above one cell per thread of a CTA, a ragged cell count
        engine("large_tissues", sets=96, cells=733, minutes=2.0, kept=True),
        # cell-ordered grids of uneven sizes (up to 48 x 48)
        engine("ordered_grids", model=GRID, sets=200, cells=48, width=8, minutes=2.0, analyses="none", kept=True),
        # the synchrony feature of a recorded generation
        {"name": "synchrony", "path": "synchrony", "sets": 1500, "samples": 600, "cells": 200},
        # ranking a pool of candidates with an ensemble, from host memory
        {"name": "rank", "path": "rank", "rows": 300000, "nets": 4},
        # predictions for inputs on the GPU, a ragged count
        {"name": "predict", "path": "predict", "rows": 100003, "inputs": 44, "outputs": 5},
        # loss and gradients of one training batch, some targets undefined
        {"name": "gradients", "path": "gradients", "rows": 4000, "inputs": 44, "outputs": 5},
        # training from new weights
        {"name": "fit", "path": "fit", "rows": 40000, "batch": 2048, "epochs": 3, "inputs": 44, "outputs": 5},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))

    path = rng.choice(["engine"] * 6 + ["grid", "grid", "synchrony", "rank", "predict", "predict", "gradients", "fit"])
    if path in ("engine", "grid"):
        if path == "grid":
            sets, cells, width = logint(1, 240), rng.randint(8, 48), 8
            area = cells * cells / 2.0
        else:
            sets, cells, width = logint(1, 2500), logint(8, 900), rng.choice([1, 4, 5])
            area = cells
        # as many steps as the largest listed case's work leaves, at most 10 minutes
        budget = 0.4 * 4096 * 200 * 3.0 * (1.0 if path == "engine" and cells <= 224 else 0.15)
        minutes = min(10.0, max(0.5, round(budget / (sets * area), 1)))
        if sets * area * minutes > budget:
            sets = max(1, int(budget / (area * minutes)))
        kept = rng.random() < 0.5
        analyses = "none" if path == "grid" else rng.choice(["none", "basic", "oscillation", "oscillation", "all"])
        return {"path": "engine", "model": GRID if path == "grid" else NETWORK, "sets": sets, "cells": cells,
                "width": width, "minutes": minutes, "bits": 32 if path == "engine" and rng.random() < 0.25 else 64,
                "analyses": analyses, "cell_params": path == "engine" and sets <= 64 and rng.random() < 0.4,
                "kept": kept}
    if path == "synchrony":
        return {"path": path, "sets": logint(20, 1500), "samples": logint(30, 600), "cells": logint(10, 200)}
    if path == "rank":
        return {"path": path, "rows": logint(1000, 300000), "nets": rng.randint(1, 4)}
    if path == "predict":
        return {"path": path, "rows": logint(1, 300000), "inputs": rng.randint(4, 64), "outputs": rng.randint(1, 8)}
    if path == "gradients":
        return {"path": path, "rows": logint(50, 16000), "inputs": rng.randint(4, 64), "outputs": rng.randint(1, 8)}
    batch = rng.choice([512, 1024, 2048, 4096])
    steps = rng.randint(2, 12)
    return {"path": "fit", "rows": batch * steps + rng.randint(0, batch - 1), "batch": batch,
            "epochs": rng.randint(1, 4), "inputs": rng.randint(4, 64), "outputs": rng.randint(2, 8)}


# --------------------------------------------------------- engine inputs


def _engine_inputs(case, seed):
    """The batch's sets as plain arrays: [(offsets, ids, params, cell
    params or None, initial concentrations or None)]."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    if case["model"] == GRID:
        # N x N grids of uneven N, up to case["cells"] a side
        sides = np.random.Generator(np.random.PCG64(case["sets"])).integers(case["width"], case["cells"] + 1,
                                                                            size=case["sets"])
        graphs = {}
        for n in sides:
            n = int(n)
            if n not in graphs:
                graphs[n] = default_graph(n * n, n)
            p = GRID_TEMPLATE * np.exp(rng.uniform(-0.15, 0.15, size=GRID_TEMPLATE.size))
            out.append(graphs[n] + (p, None, np.array([p[0] * 1.1, p[1] / p[0]])))
        return out
    off, ids = default_graph(case["cells"], case["width"])
    p0 = _network_template()
    for _ in range(case["sets"]):
        spread = 2.0 if case["sets"] > 1 else 1.1
        p = p0 * np.exp(rng.uniform(-np.log(spread), np.log(spread), size=p0.size))
        cell = p[None, :] * rng.uniform(0.95, 1.05, size=(case["cells"], p.size)) if case["cell_params"] else None
        out.append((off, ids, p, cell, None))
    return out


def _analyses(case):
    if case["model"] == GRID or case["analyses"] == "none":
        return []
    cells = case["cells"]
    basic = E.Analysis.basic(list(range(len(NETWORK_SPECIES))), 0, cells)
    if case["analyses"] == "basic":
        return [basic]
    if case["analyses"] == "oscillation":
        return [E.Analysis.oscillation([MARKER], 0, cells, 0.0, float("inf"), 4.0, INTERVAL)]
    return [basic, E.Analysis.oscillation([MARKER, NETWORK_SPECIES.index("p0")], 0, cells, 0.0, float("inf"), 4.0,
                                          INTERVAL)]


def _read_sets(count):
    """The sets whose whole state a program looks at: all of a few, a sample
    of many."""
    return range(0, count, max(1, count // 16))


def _read(case, b, analyses):
    out = {"state": [b.state(i) for i in _read_sets(case["sets"])], "status": b.status()}
    for k, a in enumerate(analyses):
        if a.kind == E.BASIC:
            r = [b.basic(k, i) for i in _read_sets(case["sets"])]
            out["basic"] = {f: np.stack([x[f] for x in r]) for f in
                            ("mins", "maxs", "sums", "cell_mins", "cell_maxs", "cell_sums")}
        elif a.kind == E.OSCILLATION:
            amps, pers = b.oscillation_all(k)
            out["amplitude"], out["period"] = amps, pers
    out["state"] = np.concatenate([s.reshape(-1) for s in out["state"]])
    return out


def _batch(state):
    case = state["case"]
    return E.Batch(state["library"], state["sets"], DT, INTERVAL, state["analyses"],
                   precision=E.FP64 if case["bits"] == 64 else E.FP32_KAHAN)


# ------------------------------------------------------ surrogate inputs


def _network_rows(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    X = rng.uniform(-1.0, 1.0, size=(case["rows"], case["inputs"])).astype(np.float32)
    A = rng.normal(size=(case["inputs"], case["outputs"])) / np.sqrt(case["inputs"])
    Y = np.tanh(2.0 * X.astype(np.float64) @ A) + 0.05 * rng.normal(size=(case["rows"], case["outputs"]))
    mask = (rng.uniform(size=Y.shape) > 0.15).astype(np.float32)
    return X, Y.astype(np.float32), mask


def _trajectories(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sets, samples, cells = case["sets"], case["samples"], case["cells"]
    t = torch.arange(samples, device="cuda", dtype=torch.float64)[None, :, None]
    phase = torch.rand((sets, 1, cells), device="cuda", dtype=torch.float64, generator=g)
    period = 40.0 + 40.0 * torch.rand((sets, 1, 1), device="cuda", dtype=torch.float64, generator=g)
    # damped, slightly out of phase across the tissue
    X = torch.sin(6.283185307179586 * t / period + 2.0 * phase)
    X.mul_(torch.exp(-t / 300.0)).mul_(25.0).add_(40.0)
    counts = torch.randint(max(2, samples - 20), samples + 1, (sets,), device="cuda", generator=g)
    return X, counts.cpu().numpy().astype(np.int32)


def _net_weights(n_in, n_out, seed):
    """Weights of a trained network's size and spread, so that predictions
    cover the outputs' range: {W: [...], b: [...]} in float32."""
    rng = np.random.Generator(np.random.PCG64(seed))
    shapes = [(surrogate.HIDDEN, surrogate.IN_PAD), (surrogate.HIDDEN, surrogate.HIDDEN),
              (surrogate.HIDDEN, surrogate.HIDDEN), (surrogate.OUT_PAD, surrogate.HIDDEN)]
    W, b = [], []
    for i, (o, n) in enumerate(shapes):
        w = np.zeros((o, n), np.float32)
        rows, cols = (o if i < 3 else n_out), (n if i > 0 else n_in)
        w[:rows, :cols] = rng.normal(0.0, np.sqrt(2.0 / cols), size=(rows, cols))
        c = np.zeros(o, np.float32)
        c[:rows] = rng.normal(0.0, 0.1, size=rows)
        W.append(w)
        b.append(c)
    return W, b


def _net(n_in, n_out, seed):
    net = surrogate.MLP(n_in, n_out, seed=0)
    W, b = _net_weights(n_in, n_out, seed)
    for i in range(4):
        net.W[i].copy_(torch.from_numpy(W[i]))
        net.b[i].copy_(torch.from_numpy(b[i]))
    return net


# ------------------------------------------------------- prepare and run


def prepare(case, seed):
    state = {"case": case}
    path = case["path"]
    if path == "engine":
        state["library"] = _library(case["model"])
        state["sets"] = [E.ParameterSet(off, ids, p, cell_params=cell, init_conc=ic, duration=case["minutes"])
                         for off, ids, p, cell, ic in _engine_inputs(case, seed)]
        state["analyses"] = _analyses(case)
        if case["kept"]:
            state["batch"] = _batch(state)
    elif path == "synchrony":
        state["X"], state["counts"] = _trajectories(case, seed)
    elif path == "rank":
        n = len(search.active_params())
        nets = [_net(n, 5, 100 * seed + i) for i in range(case["nets"])]
        state["net"] = search.Surrogate(nets, mu=[3.3, 3.9, 0.2, 0.0, 0.0], sd=[0.4, 0.8, 0.3, 1.0, 1.0])
        state["P"] = search.draw_candidates(case["rows"], seed)
    elif path == "predict":
        X, _, _ = _network_rows(case, seed)
        state["net"] = _net(case["inputs"], case["outputs"], seed)
        state["X"] = torch.from_numpy(X).cuda()
    elif path == "gradients":
        state["X"], state["T"], state["mask"] = _network_rows(case, seed)
        state["net"] = _net(case["inputs"], case["outputs"], seed)
    else:
        state["X"], state["T"], state["mask"] = _network_rows(case, seed)
        state["seed"] = seed
    return state


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "engine":
        if case["kept"]:
            b = state["batch"]
            b.reset()
            b.run()
            return _read(case, b, state["analyses"])
        b = _batch(state)
        b.run()
        out = _read(case, b, state["analyses"])
        b.close()
        return out
    if path == "synchrony":
        return search.synchrony_batch(state["X"], state["counts"])
    if path == "rank":
        return search.score_candidates(state["net"], state["P"])
    if path == "predict":
        return state["net"].predict_device(state["X"])
    if path == "gradients":
        loss, dW, db = state["net"].gradients(state["X"], state["T"], state["mask"])
        return {"loss": loss, "dW": dW, "db": db}
    net = surrogate.MLP(case["inputs"], case["outputs"], seed=state["seed"], lr=2e-4)
    losses = net.fit(state["X"], state["T"], state["mask"], epochs=case["epochs"], batch=case["batch"],
                     seed=state["seed"])
    return {"losses": np.array(losses, np.float32), "W": net.W, "b": net.b}


# ------------------------------------------------------------------- work


def _layer_flops(n_in, n_out):
    return 2.0 * (n_in * surrogate.HIDDEN + 2 * surrogate.HIDDEN ** 2 + surrogate.HIDDEN * n_out)


# floating operations of one cell-step: rates and neighbour averages (four
# and a half neighbours), two per delta term, two per species
NETWORK_FLOPS = 57.0 + 2 * 5.5 + 2 * sum(len(r[3]) for r in NETWORK_REACTIONS) + 2 * len(NETWORK_SPECIES)
GRID_FLOPS = 9.0 + 2 * 5.5 + 2 * sum(len(r[3]) for r in GRID_REACTIONS) + 2 * len(GRID_SPECIES)


def work(case):
    path = case["path"]
    if path == "engine":
        if case["model"] == GRID:
            lo, hi = case["width"], case["cells"]
            cells = case["sets"] * sum(n * n for n in range(lo, hi + 1)) / float(hi - lo + 1)
            params, nsp, flops = GRID_TEMPLATE.size, 2, GRID_FLOPS
        else:
            cells = case["sets"] * case["cells"]
            params, nsp, flops = _network_template().size, len(NETWORK_SPECIES), NETWORK_FLOPS
        steps = int(np.ceil(case["minutes"] / INTERVAL)) * int(INTERVAL / DT)
        rows = cells if case["cell_params"] else case["sets"]
        nbytes = 8.0 * (rows * params + cells * nsp)
        return {"bytes": nbytes, "flops": cells * steps * flops}
    if path == "synchrony":
        n = float(case["sets"]) * case["samples"] * case["cells"]
        return {"bytes": 8.0 * n, "flops": 6.0 * n}
    if path == "rank":
        n = case["rows"]
        return {"bytes": 8.0 * n * (len(workloads.template_params()) + 1),
                "flops": case["nets"] * n * _layer_flops(len(search.active_params()), 5)}
    n_in, n_out, n = case["inputs"], case["outputs"], case["rows"]
    weights = 4.0 * (n_in * surrogate.HIDDEN + 2 * surrogate.HIDDEN ** 2 + surrogate.HIDDEN * n_out)
    if path == "predict":
        return {"bytes": 4.0 * n * (n_in + n_out) + weights, "flops": n * _layer_flops(n_in, n_out)}
    if path == "gradients":
        return {"bytes": 4.0 * n * (n_in + 2 * n_out) + 2 * weights, "flops": 3.0 * n * _layer_flops(n_in, n_out)}
    steps = case["epochs"] * (n // case["batch"])
    return {"bytes": 4.0 * n * (n_in + 2 * n_out) + steps * 6 * weights,
            "flops": 3.0 * steps * case["batch"] * _layer_flops(n_in, n_out)}


# ------------------------------------------------------------------ exact


def _joined(sets, dev):
    """The sets' cells in one index space: padded neighbour ids, counts."""
    total = sum(len(s[0]) - 1 for s in sets)
    degree = max(int(np.diff(s[0]).max()) for s in sets)
    nbr = np.zeros((total, degree), np.int64)
    has = np.zeros((total, degree), bool)
    base = 0
    for off, ids, _, _, _ in sets:
        n = len(off) - 1
        count = np.diff(off)
        for j in range(degree):
            on = count > j
            nbr[base:base + n][on, j] = ids[off[:-1][on] + j] + base
            has[base:base + n, j] = on
        base += n
    return torch.from_numpy(nbr).to(dev), torch.from_numpy(has).to(dev)


def _network_exact(case, sets, dev):
    nbr, has = _joined(sets, dev)
    n = nbr.shape[0]
    count = has.sum(1).double()
    P = np.concatenate([np.repeat(p[None], len(off) - 1, 0) if cell is None else cell
                        for off, _, p, cell, _ in sets])
    P = torch.from_numpy(np.ascontiguousarray(P.T)).to(dev)
    names = [r[0] for r in NETWORK_REACTIONS]
    rate = {r: P[i] for i, r in enumerate(names)}
    delay = {r: P[len(names) + i].long() for i, r in enumerate(NETWORK_DELAYED)}
    crit = {s: P[len(names) + len(NETWORK_DELAYED) + i] for i, s in enumerate(NETWORK_CRITICAL)}
    deep = int(max(d.max() for d in delay.values())) + 2
    keep = ["m%d" % g for g in range(GENES)] + ["d%d" % g for g in range(GENES)] + ["ms", "ps"]
    hist = {s: torch.zeros((deep, n), dtype=torch.float64, device=dev) for s in keep}
    cells = torch.arange(n, device=dev)
    x = {s: torch.zeros(n, dtype=torch.float64, device=dev) for s in NETWORK_SPECIES}
    steps = int(np.ceil(case["minutes"] / INTERVAL)) * int(INTERVAL / DT)

    def past(s, r, t):  # own reads: delay k is lag k - 1
        return hist[s].view(-1)[((t - (delay[r] - 1)) % deep) * n + cells]

    def around(s, r, t):  # neighbour reads: the row of lag k, each at the neighbour's place
        rows = ((t - delay[r]) % deep)[:, None] * n + nbr
        return torch.where(has, hist[s].view(-1)[rows], 0.0).sum(1) / count

    for t in range(steps):
        for s in keep:
            hist[s][t % deep] = x[s]
        r = {}
        for g in range(GENES):
            up = "d%d" % REPRESSOR[g]
            f = past(up, "msyn%d" % g, t) / crit[up]
            act = 1.0
            if g < 2:
                act = 1.0 + around("ps", "msyn%d" % g, t) / crit["ps"]
            r["msyn%d" % g] = rate["msyn%d" % g] * act / (act + f * f)
            m, p, d = x["m%d" % g], x["p%d" % g], x["d%d" % g]
            r["mdeg%d" % g] = rate["mdeg%d" % g] * m
            r["psyn%d" % g] = rate["psyn%d" % g] * past("m%d" % g, "psyn%d" % g, t)
            r["pdeg%d" % g] = rate["pdeg%d" % g] * p
            r["bind%d" % g] = rate["bind%d" % g] * p * p
            r["dis%d" % g] = rate["dis%d" % g] * d
            r["ddeg%d" % g] = rate["ddeg%d" % g] * d
        f = past("d0", "mssyn", t) / crit["d0"]
        r["mssyn"] = rate["mssyn"] / (1.0 + f * f)
        r["msdeg"] = rate["msdeg"] * x["ms"]
        r["pssyn"] = rate["pssyn"] * past("ms", "pssyn", t)
        r["psdeg"] = rate["psdeg"] * x["ps"]
        new = {}
        for s in NETWORK_SPECIES:
            change = sum(delta[s] * r[name] for name, _, _, delta in NETWORK_REACTIONS if s in delta)
            new[s] = x[s] + DT * change
        x = new
    return torch.stack([x[s] for s in NETWORK_SPECIES])


def _grid_exact(case, sets, dev):
    nbr, has = _joined(sets, dev)
    n = nbr.shape[0]
    count = has.sum(1).double()
    P = torch.from_numpy(np.concatenate([np.repeat(s[2][None], len(s[0]) - 1, 0) for s in sets])).to(dev).T
    x = torch.from_numpy(np.concatenate([np.repeat(s[4][None], len(s[0]) - 1, 0) for s in sets])).to(dev).T.contiguous()
    # a cell may be updated once its lower-numbered neighbours are; level by
    # level that is the cell order
    level = torch.zeros(n, dtype=torch.long, device=dev)
    lower = has & (nbr < torch.arange(n, device=dev)[:, None])
    while True:
        up = torch.where(lower, level[nbr] + 1, 0).amax(1)
        if torch.equal(up, level):
            break
        level = up
    levels = [torch.nonzero(level == l)[:, 0] for l in range(int(level.max()) + 1)]
    levels = [(c, nbr[c], has[c], lower[c], count[c], P[:, c]) for c in levels]
    steps = int(np.ceil(case["minutes"] / INTERVAL)) * int(INTERVAL / DT)
    before = x.clone()  # the row of one step back, which the new values replace cell by cell
    for _ in range(steps):
        row = torch.empty_like(x)
        for c, nb, on, low, cnt, p in levels:
            avg = torch.where(low, row[:, nb], torch.where(on, before[:, nb], 0.0)).sum(2) / cnt
            u, v = x[0, c], x[1, c]
            conv, turn = p[1] * u, p[2] * u * u * v
            du = p[0] - conv + turn - p[3] * u + p[4] * (avg[0] - u)
            dv = conv - turn + p[5] * (avg[1] - v)
            row[:, c] = torch.stack([u + DT * du, v + DT * dv])
        before, x = x, row
    return x


def _per_set_state(state, sets, chosen):
    """[species][joined cells] as the concatenated [species][cells] of the
    chosen sets."""
    start = np.concatenate([[0], np.cumsum([len(s[0]) - 1 for s in sets])])
    return torch.cat([state[:, start[i]:start[i + 1]].reshape(-1) for i in chosen])


def _synchrony_exact(X):
    """[sets][samples][cells] -> mean pairwise Pearson correlation."""
    z = X - X.mean(1, keepdim=True)
    z = z / z.norm(dim=1, keepdim=True)
    n = X.shape[2]
    return (z.sum(2).square().sum(1) - n) / (n * (n - 1.0))


def _net_exact(W, b, X, n_in, n_out):
    h = X
    for i in range(3):
        z = h @ W[i][:, :h.shape[1]].T + b[i]
        h = 0.5 * z * (1.0 + torch.erf(z * 0.7071067811865476))
    return h @ W[3][:n_out].T + b[3][:n_out]


def exact(case, seed):
    path = case["path"]
    dev = torch.device("cuda")
    if path == "engine":
        sets = _engine_inputs(case, seed)
        if case["model"] == GRID:
            if case["minutes"] > 3.0:
                return None
            x = _grid_exact(case, sets, dev)
            return {"state": _per_set_state(x, sets, _read_sets(case["sets"])), "status": None}
        state = _network_exact(case, sets, dev)
        return {"state": _per_set_state(state, sets, _read_sets(case["sets"]))}
    if path == "synchrony":
        X, counts = _trajectories(case, seed)
        return torch.stack([_synchrony_exact(X[i:i + 1, :int(k)])[0] for i, k in enumerate(counts)])
    if path == "rank":
        P = torch.from_numpy(search.draw_candidates(case["rows"], seed)).to(dev)
        idx = torch.from_numpy(search.active_params()).to(dev)
        t = torch.from_numpy(search.template()).to(dev)[idx]
        X = torch.log(P[:, idx] / t) / float(np.log(search.SPREAD))
        y = 0.0
        for i in range(case["nets"]):
            W, b = _net_weights(len(idx), 5, 100 * seed + i)
            W, b = [torch.from_numpy(w).to(dev).double() for w in W], [torch.from_numpy(v).to(dev).double() for v in b]
            y = y + torch.cat([_net_exact(W, b, x, len(idx), 5) for x in X.split(65536)])
        y = y / case["nets"]
        y = y * torch.tensor([0.4, 0.8, 0.3, 1.0, 1.0], device=dev, dtype=torch.float64)
        y = y + torch.tensor([3.3, 3.9, 0.2, 0.0, 0.0], device=dev, dtype=torch.float64)
        per = torch.exp(y[:, 0].clamp(-10.0, 10.0))
        amp = ((y[:, 1] - float(np.log(search.AMP_MIN))) / search.AMP_RAMP + 0.5).clamp(0.0, 1.0)
        region = -(per - search.TARGET_PERIOD).abs() / search.PERIOD_TOL + 0.5 * amp + 0.5 * y[:, 3].clamp(0.0, 1.0)
        return y[:, 4] + search.REGION_WEIGHT * region
    if path == "fit":
        return None
    X, T, mask = _network_rows(case, seed)
    W, b = _net_weights(case["inputs"], case["outputs"], seed)
    W, b = [torch.from_numpy(w).to(dev).double() for w in W], [torch.from_numpy(v).to(dev).double() for v in b]
    X = torch.from_numpy(X).to(dev).double()
    if path == "predict":
        return torch.cat([_net_exact(W, b, x, case["inputs"], case["outputs"]) for x in X.split(65536)])
    T, mask = torch.from_numpy(T).to(dev).double(), torch.from_numpy(mask).to(dev).double()
    for w in W + b:
        w.requires_grad_(True)
    y = _net_exact(W, b, X, case["inputs"], case["outputs"])
    loss = (mask * (y - T).square()).sum() / mask.sum()
    g = torch.autograd.grad(loss, W + b)
    return {"loss": loss.detach(), "dW": list(g[:4]), "db": list(g[4:])}
