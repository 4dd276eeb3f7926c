"""The synchrony kernel at the edges of its thread groups, its blocks of
eight samples, its CTA sizes and its clusters, against a float64 numpy
two-pass reference.  Both sum at most a few thousand correlation products
of magnitude <= 1 per pair, so they agree to 1e-12."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traces(sets, samples, cells, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    t = np.arange(samples)[None, :, None]
    X = 40.0 + 25.0 * np.sin(0.13 * t + rng.uniform(0, 2, size=(sets, 1, cells))) + rng.normal(size=(sets, samples, cells))
    return np.ascontiguousarray(X)


def _check(X, counts, view=None):
    import torch
    from dense_b200.search import synchrony, synchrony_batch
    T = torch.tensor(X, device="cuda") if view is None else view
    got = synchrony_batch(T, np.asarray(counts, np.int32))
    for i, k in enumerate(counts):
        want = synchrony(X[i, :k]) if k > 0 else float("nan")
        assert (np.isnan(want) and np.isnan(got[i])) or abs(got[i] - want) < 1e-12, (i, k, got[i], want)


@pytest.mark.parametrize("cells", [1, 2, 31, 32, 33, 64, 65, 129, 256, 257, 513, 1023, 1024])
def test_cell_counts(cells):
    _check(_traces(3, 70, cells, cells), [70, 33, 8])


@pytest.mark.parametrize("samples", [1, 2, 7, 8, 9, 15, 16, 17, 63, 64, 65, 511, 1300])
def test_sample_counts(samples):
    _check(_traces(4, samples, 40, samples), [samples, max(0, samples - 1), samples // 2, 0])


@pytest.mark.parametrize("sets,samples,cells", [(1, 2000, 200), (400, 60, 20), (297, 120, 150)])
def test_cluster_and_thread_rules(sets, samples, cells):
    _check(_traces(sets, samples, cells, sets), [samples - (i % 5) for i in range(sets)])


def test_layouts_and_special_values():
    import torch
    X = _traces(5, 90, 36, 9)
    X[1, :, 4] = 7.0        # a constant cell
    X[2, 50, 3] = np.inf    # no cell counts
    X[3, 89, 35] = np.nan
    counts = [90, 90, 90, 90, 41]
    with np.errstate(invalid="ignore"):
        _check(X, counts)
        outer = torch.tensor(np.ascontiguousarray(X.transpose(1, 0, 2)), device="cuda").transpose(0, 1)
        _check(X, counts, outer)  # the samples outside the sets
        wide = torch.full((5, 90, 3, 37), float("nan"), dtype=torch.float64, device="cuda")
        wide[:, :, 1, :36] = torch.tensor(X, device="cuda")
        _check(X, counts, wide[:, :, 1, :36])  # odd strides
