"""The synchrony kernel on traces whose squares leave the range of float64,
and on cells at the threshold of a constant trace, against the float64 numpy
two-pass reference."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traces(samples, cells, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    t = np.arange(samples)[:, None]
    return 3.0 + np.sin(0.2 * t + rng.uniform(0, 2, size=(1, cells))) + 0.1 * rng.normal(size=(samples, cells))


def _check(X, tolerance=1e-12):
    import torch
    from dense_b200.search import synchrony, synchrony_batch
    with np.errstate(over="ignore"):
        want = [synchrony(x) for x in X]
    got = synchrony_batch(torch.tensor(X, device="cuda"), np.full(len(X), X.shape[1], np.int32))
    for g, w in zip(got, want):
        assert abs(g - w) < tolerance, (g, w)


@pytest.mark.parametrize("samples", [3, 7, 8, 9, 64, 130, 1300])
@pytest.mark.parametrize("mean,spread", [(2e154, 1e152), (-3e200, 3e198), (1e160, 1e160), (1e300, 1e298)])
def test_squares_out_of_range(mean, spread, samples):
    """Means whose square is not a float64, and deviations whose square is
    not (norms of infinity: every quotient is 0).  A mean of m rounds to
    eps m, so a unit trace is known to eps m / spread."""
    X = np.stack([mean + spread * _traces(samples, 24, i) for i in range(3)])
    _check(X, 1e-12 + 8 * 2.2e-16 * abs(mean) / spread)


@pytest.mark.parametrize("cells", [3, 40, 700])
@pytest.mark.parametrize("samples", [16, 600])
@pytest.mark.parametrize("above", [False, True])
def test_cells_next_to_the_threshold(above, samples, cells):
    """A cell counts when its norm is above 1e-12 (1 + the largest magnitude),
    the whole of it: a magnitude's lower word moves the threshold by up to a
    millionth."""
    X = np.stack([_traces(samples, cells, i) for i in range(2)])
    X[1, samples // 2, 2] = np.nextafter(4.0e6, 0.0)  # its lower word is all ones
    top = np.abs(X[1]).max()
    short = np.array(np.array(top).view(np.uint64) & np.uint64(0xFFFFFFFF00000000)).view(np.float64)[()]
    assert top > short
    norm = 1e-12 * (1.0 + (top * (1 + 1e-8) if above else 0.5 * (top + short)))
    half = norm / np.sqrt(samples)
    X[1, :, 0] = np.where(np.arange(samples) % 2, half, -half)
    _check(X)
