"""Kernel attributes are set on every device that a process uses
(csrc/engine/per_device.hpp, compiled for the host), and the step kernels'
launchers go through it."""

import os
import re
import subprocess

from tests.conftest import ROOT

ENGINE = os.path.join(ROOT, "dense_b200", "csrc", "engine")


def test_set_up_runs_once_on_each_device(tmp_path):
    exe = str(tmp_path / "per_device_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", ENGINE,
                    os.path.join(ROOT, "tests", "native", "per_device_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_launchers_keep_no_flag_for_all_devices():
    with open(os.path.join(ENGINE, "step_kernel.cuh")) as f:
        src = f.read()
    assert not re.search(r"static (bool|int) \w+ = (false|0);", src)
    for variant in ("STEP", "CLUSTER"):
        body = src[src.index("#define DENSE_B200_%s_VARIANT" % variant):]
        assert "opt_in<k>(" in body[:body.index("\n  }\n")]
