"""Runs host code of the engine on a machine without a GPU: a program in a
process of its own with tests/native/fake_cudart.c in front of the CUDA
runtime, and the calls it made."""

import os
import subprocess
import sys
import tempfile

from tests.conftest import ROOT

_built = []


def _library():
    if not _built:
        out = os.path.join(tempfile.mkdtemp(prefix="fake_cudart_"), "libfake_cudart.so")
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-I", os.path.join(cuda, "include"),
                        os.path.join(ROOT, "tests", "native", "fake_cudart.c"), "-o", out], check=True)
        _built.append(out)
    return _built[0]


def calls(program, tmp_path, **env):
    """The lines of the call log of a Python program; `env` adds to its
    environment (FAKE_CAPACITY, FAKE_CLUSTERS)."""
    log = str(tmp_path / "calls.log")
    if os.path.exists(log):
        os.remove(log)
    e = dict(os.environ, LD_PRELOAD=_library(), FAKE_CUDART_LOG=log, CUDA_VISIBLE_DEVICES="",
             PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    e.update({k: str(v) for k, v in env.items()})
    r = subprocess.run([sys.executable, "-c", program], env=e, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    with open(log) as f:
        return f.read().splitlines()
