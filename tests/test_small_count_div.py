"""The short division by a neighbour count (csrc/engine/count_div.cuh),
compiled for the host and compared with IEEE division."""

import os
import subprocess

from tests.conftest import ROOT


def test_small_count_division_is_ieee_division(tmp_path):
    exe = str(tmp_path / "small_count_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "dense_b200", "csrc", "engine"),
                    os.path.join(ROOT, "tests", "native", "small_count_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
