"""MLP.forward, the network a GEMM a layer: its outputs are the whole-network
kernel's to rounding, and the layers' outputs are left in Z and H."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [128, 384])
def test_forward_agrees_with_predictions(rows):
    import torch
    from dense_b200.surrogate import IN_PAD, MLP, OUT_PAD
    net = MLP(40, 6, seed=3)
    for b in net.b:
        b.uniform_(-0.1, 0.1)
    X = torch.from_numpy(np.random.Generator(np.random.PCG64(1)).uniform(-1, 1, size=(rows, 40)).astype(np.float32)).cuda()
    Xb = torch.zeros((rows, IN_PAD), dtype=torch.bfloat16, device="cuda")
    Xb[:, :40] = X.to(torch.bfloat16)
    Y = net.forward(Xb)
    net.k.check()
    assert Y.shape == (rows, OUT_PAD) and len(net.Z) == 3 and len(net.H) == 4
    want = net.predict_device(X)
    # the products' sums run in another order: a BF16 rounding of an
    # activation may fall the other way
    assert torch.linalg.norm(Y[:, :6] - want) < 1e-2 * torch.linalg.norm(want)
    # H is GELU(Z) in BF16 (an ulp is at most 2^-7 of the value)
    assert torch.allclose(torch.nn.functional.gelu(net.Z[0]), net.H[1].float(), rtol=0.01, atol=1e-6)
    # new weights are taken at once
    net.W[3].zero_()
    assert torch.equal(net.forward(Xb)[:, :6], net.b[3][:6].expand(rows, 6))
