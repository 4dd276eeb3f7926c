"""The register kernel's row table (in static shared memory) leaves room for
the largest dynamic share of a CTA in models with many reactions: such a model
forms its rows per read, as before there was a table, and its kernels can be
opted in to that share."""

import os
import subprocess

import pytest

from tests import network_model as N
from tests.conftest import ROOT


def _model(species, delays, reactions):
    names = ["s%d" % i for i in range(species)]
    out = [("d%d" % i, True, "return c.getCon(s%d, c.getDelay(dreact_d%d));" % (i % species, i), {"s0": 1})
           for i in range(delays)]
    return names, [], out + [("r%d" % i, False, "return c.getRate(r%d) * c.getCon(s%d);" % (i, i % species), {"s0": -1})
                             for i in range(reactions - delays)]


def _write(model, folder):
    for f, lines in N.cases._headers(*model).items():
        (folder / f).write_text("\n".join(lines) + "\n")


@pytest.mark.parametrize("species,delays,reactions,table", [
    (14, 10, 32, True), (24, 16, 60, True), (25, 16, 60, False), (32, 12, 500, True), (32, 12, 700, False),
    (32, 12, 2000, False), (2, 0, 6, False)])
def test_table_only_where_it_fits(species, delays, reactions, table, tmp_path):
    _write(_model(species, delays, reactions), tmp_path)
    engine, api = (os.path.join(ROOT, "dense_b200", "csrc", d) for d in ("engine", "model_api"))
    exe = str(tmp_path / "static_smem")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-w", "-I", api, "-I", str(tmp_path), "-I", engine, "-I",
                    os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "native", "static_smem.cpp"), "-o", exe],
                   check=True)
    has, static, dynamic, most = map(int, subprocess.run([exe], capture_output=True, text=True).stdout.split())
    assert bool(has) == table
    assert static + dynamic <= most
