"""Weight gradients of batches of more rows than 74 (output layer: 148) ranges
of four 64-row blocks: summed over the same ranges as a layer at a time, so
equal to it bit for bit, and no further from the float64 products of the same
BF16 operands."""

import numpy as np
import pytest

from tests.test_chain_gpu import _layered, _net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out", [5, 70])
@pytest.mark.parametrize("rows", [4097, 5376, 5377, 9000, 18944, 19200, 38400, 60001])
def test_gradients_equal_the_layered_pass(rows, n_out):
    import torch
    net = _net(44, n_out, 1)
    rng = np.random.Generator(np.random.PCG64(rows))
    X = rng.uniform(-1, 1, size=(rows, 44)).astype(np.float32)
    T = rng.normal(size=(rows, n_out)).astype(np.float32)
    mask = (rng.uniform(size=T.shape) > 0.3).astype(np.float32)
    _, dW, db = _layered(net, *(torch.tensor(v, device="cuda") for v in (X, T, mask)))
    _, gW, gb = net.gradients(X, T, mask)
    for i in range(4):
        assert torch.equal(gW[i], dW[i]) and torch.equal(gb[i], db[i]), i
