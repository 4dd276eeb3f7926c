"""Tests of DENSE's own models on a machine without a DENSE tree: skipped, and
failed where the tree is there."""

import pytest
from torch.multiprocessing import ProcessRaisedException

from dense_b200.models import ENV, MissingModelError, model_dir
from tests import conftest


class _Outcome:
    def __init__(self, error):
        self.exception = self.forced = error

    def force_exception(self, error):
        self.forced = error


@pytest.mark.parametrize("error,skips", [
    (MissingModelError("model directory x not found"), True),
    (ProcessRaisedException("dense_b200.models.MissingModelError: x", 1, 2), True),
    (ProcessRaisedException("AssertionError", 1, 2), False),
    (RuntimeError("nvcc failed"), False),
    (AssertionError("a program's output: dense_b200.models.MissingModelError: x"), False),
    (None, False)])
@pytest.mark.parametrize("tree", [None, "empty", "dense"])
def test_missing_models(error, skips, tree, tmp_path, monkeypatch):
    monkeypatch.delenv(ENV, raising=False)
    if tree:
        monkeypatch.setenv(ENV, str(tmp_path))
    if tree == "dense":
        (tmp_path / "models").mkdir()
    out = _Outcome(error)
    conftest._skip_without_tree(out)
    assert isinstance(out.forced, pytest.skip.Exception) == (skips and tree != "dense")
    assert out.exception is error


def test_an_unnamed_tree_is_a_missing_model(monkeypatch):
    monkeypatch.delenv(ENV, raising=False)
    with pytest.raises(MissingModelError, match=ENV):
        model_dir("her_model_2014")
