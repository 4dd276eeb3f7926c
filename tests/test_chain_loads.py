"""Kernels that are resident while the one before them still writes their
inputs (programmatic dependent launch, `follow_previous`) read global memory
with plain loads: a `__restrict__` pointer to const, `__ldg` or a
cache-hinted load may be moved above the wait by the compiler."""

import os
import re

from tests.conftest import ROOT


def test_dependent_kernels_use_plain_loads():
    with open(os.path.join(ROOT, "dense_b200", "csrc", "surrogate", "chain.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    kernels = [m.start() for m in re.finditer(r"__global__", src)]
    checked = 0
    for a in kernels:
        body = src[a:src.index("\n}\n", a)]
        if "follow_previous();" not in body:
            continue
        checked += 1
        assert not re.search(r"__restrict__|__ldg\(|__ldc[a-z]\(|__ldlu\(|ld\.global\.nc", body), body[:120]
    assert checked == 5
