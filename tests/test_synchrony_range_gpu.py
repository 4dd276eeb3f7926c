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
