"""bench.py's reference arm where DENSE is not on the machine."""

import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("tree", [None, "empty"])
def test_reference_arm_says_that_it_is_unavailable(tree, tmp_path):
    from oracle.build import oracle_lib_path, ref_lib_path
    if os.path.exists(ref_lib_path("her_model_2014")) or os.path.exists(oracle_lib_path("her_model_2014")):
        pytest.skip("DENSE's model was built here")
    env = {k: v for k, v in os.environ.items() if k != "DENSE_REF_DIR"}
    if tree:
        env["DENSE_REF_DIR"] = str(tmp_path)
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "1"], capture_output=True, text=True, timeout=300, cwd=ROOT, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout.strip())
    assert set(d) == {"impl", "unavailable"} and d["impl"] == "reference" and "\n" not in d["unavailable"]
