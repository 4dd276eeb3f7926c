"""The training pass on rows chosen by an index list with the scale of the loss
on the device (what an epoch's steps are), against a layer at a time on the
gathered rows, bit for bit; the library's gather and device-scaled loss kernels
give that pass its inputs and its output gradient."""

import numpy as np
import pytest

from tests.test_chain_gpu import _layered, _net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out", [5, 17, 70])
@pytest.mark.parametrize("rows", [1, 128, 1000, 2048, 4500])
def test_indexed_rows(rows, n_out):
    import torch
    from dense_b200.surrogate import IN_PAD, OUT_PAD
    net = _net(44, n_out, rows + n_out)
    k = net.k
    g = torch.Generator(device="cuda").manual_seed(rows)
    X = torch.rand((3000, 44), device="cuda", generator=g) * 2 - 1
    T = torch.randn((3000, n_out), device="cuda", generator=g)
    M = (torch.rand((3000, n_out), device="cuda", generator=g) > 0.3).float()
    idx = torch.randint(0, 3000, (rows,), device="cuda", generator=g).to(torch.int32)  # some rows twice
    M[idx[0].long(), 0] = 1.0

    Bp = (rows + 127) // 128 * 128
    Xb = torch.empty((Bp, IN_PAD), dtype=torch.bfloat16, device="cuda")
    Tb, Mb = torch.empty((Bp, n_out), device="cuda"), torch.empty((Bp, n_out), device="cuda")
    k.gather(X, T, M, idx, Xb, Tb, Mb)
    at = idx.long()
    assert torch.equal(Xb[:rows, :44], X[at].to(torch.bfloat16)) and torch.equal(Tb[:rows], T[at])
    assert torch.equal(Mb[:rows], M[at]) and not Mb[rows:].any() and not Xb[:, 44:].any()

    loss, dW, db = _layered(net, X[at], T[at], M[at])
    inv = torch.tensor([1.0 / max(1.0, float(M[at].sum().item()))], device="cuda")
    got = torch.zeros(1, device="cuda")
    gW, gb = net._grads()
    work = net._work(rows)
    k.train_pass(X, T, M, idx, rows, net._pack(backward=True), net.b, inv, got, work)
    k.train_finish(work, rows, n_out, gW, gb)
    # the same output gradient from the loss kernel with the scale on the device
    Y = net.forward(Xb)
    dY, dYb = torch.empty((Bp, OUT_PAD), device="cuda"), torch.empty((Bp, OUT_PAD), dtype=torch.bfloat16, device="cuda")
    dev_loss = torch.zeros(1, device="cuda")
    k.mse_dev(Y, Tb, Mb, inv, dY, dYb, dev_loss)
    k.check()
    for i in range(4):
        assert torch.equal(gW[i], dW[i]) and torch.equal(gb[i], db[i]), i
    # sums of up to a few hundred thousand float32 terms in another order
    assert abs(float(got) - loss) <= 1e-5 * abs(loss) and abs(float(dev_loss) - loss) <= 1e-5 * abs(loss)
    want = torch.empty_like(db[3])
    k.colsum(dY, want)
    assert torch.equal(want, db[3])
