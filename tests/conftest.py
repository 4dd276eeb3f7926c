import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    # the DENSE tree the fixtures and model builds read, when one is present
    from oracle.build import use_default_tree
    use_default_tree()
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200)")


def gpu_available():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if gpu_available():
        return
    skip = pytest.mark.skip(reason="no CUDA GPU")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


def _skip_without_tree(outcome):
    """Tests of DENSE's own models need its headers, or libraries built from
    them before.  On a machine with neither they are skipped, and those of
    the models written out in tests/ run; with a DENSE tree a model that is
    missing fails its test."""
    from dense_b200.models import ENV, MissingModelError
    tree = os.environ.get(ENV)
    error = outcome.exception
    # (a rank of its own process reports the error in its traceback)
    rank = type(error).__name__ == "ProcessRaisedException"
    missing = isinstance(error, MissingModelError) or (rank and "models.MissingModelError: " in str(error))
    if missing and not (tree and os.path.isdir(os.path.join(tree, "models"))):
        outcome.force_exception(pytest.skip.Exception(str(error)))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_setup(item):
    _skip_without_tree((yield))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    _skip_without_tree((yield))
