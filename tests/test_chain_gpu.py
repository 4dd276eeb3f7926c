"""The whole-network kernels (csrc/surrogate/chain.cu) against the same passes
made a layer at a time with the library's GEMM, GELU, loss, transpose and
column-sum kernels: the products accumulate in the same order, so
predictions, weight gradients (up to 4096 rows: the same row ranges) and
bias gradients are equal bit for bit; the loss is a sum in another order
(float32, a few thousand terms: 1e-5).  Sizes at the edges of the row tiles,
the 16- and 64-column output blocks and the padded inputs, and more tiles
than SMs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net(n_in, n_out, seed):
    import torch
    from dense_b200.surrogate import MLP
    net = MLP(n_in, n_out, seed=seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    for i, b in enumerate(net.b):
        b.copy_(0.2 * torch.randn(b.shape, device="cuda", generator=g))
    net.b[3][n_out:] = 0
    return net


def _layered(net, X, T=None, mask=None):
    """Outputs (and loss, dW, db) a layer at a time."""
    import torch
    from dense_b200.surrogate import EPI_BIAS, EPI_BIAS_GELU, HIDDEN, IN_PAD, OUT_PAD
    k, bf = net.k, torch.bfloat16
    B, Bp = X.shape[0], (X.shape[0] + 127) // 128 * 128
    new = lambda *s, dtype=torch.float32: torch.empty(s, dtype=dtype, device="cuda")  # noqa: E731
    Wb = [new(*w.shape, dtype=bf) for w in net.W]
    WTb = [new(w.shape[1], w.shape[0], dtype=bf) for w in net.W]
    for i, w in enumerate(net.W):
        k.cast(w, Wb[i])
        k.cast(w, WTb[i], transpose=True)
    Xb = torch.zeros((Bp, IN_PAD), dtype=bf, device="cuda")
    Xb[:B, :net.n_in] = X.to(bf)
    H, Z = [Xb], []
    for i in range(3):
        Z.append(new(Bp, HIDDEN))
        H.append(new(Bp, HIDDEN, dtype=bf))
        k.gemm(H[i], Wb[i], Z[i], EPI_BIAS_GELU, net.b[i], H[i + 1])
    Y = new(Bp, OUT_PAD)
    k.gemm(H[3], Wb[3], Y, EPI_BIAS, net.b[3])
    if T is None:
        k.check()
        return Y[:B, :net.n_out]
    Tp, Mp = torch.zeros((Bp, net.n_out), device="cuda"), torch.zeros((Bp, net.n_out), device="cuda")
    Tp[:B], Mp[:B] = T, mask
    loss, dZ, dZb = torch.zeros(1, device="cuda"), new(Bp, OUT_PAD), new(Bp, OUT_PAD, dtype=bf)
    k.mse(Y, Tp, Mp, dZ, dZb, loss)
    dW, db = [None] * 4, [None] * 4
    for i in (3, 2, 1, 0):
        rows = net.W[i].shape[0]
        dZT, HT = new(rows, Bp, dtype=bf), new(net.W[i].shape[1], Bp, dtype=bf)
        k.transpose(dZb, dZT)
        k.transpose(H[i], HT)
        dW[i], db[i] = new(*net.W[i].shape), new(rows)
        k.gemm(dZT, HT, dW[i])
        k.colsum(dZ, db[i])
        if i:
            dH, ndZ, ndZb = new(Bp, HIDDEN), new(Bp, HIDDEN), new(Bp, HIDDEN, dtype=bf)
            k.gemm(dZb, WTb[i], dH)
            k.gelu_backward(dH, Z[i - 1], ndZ, ndZb)
            dZ, dZb = ndZ, ndZb
    k.check()
    return float(loss.item()), dW, db


@pytest.mark.parametrize("rows,n_in,n_out", [(1, 44, 5), (127, 1, 1), (128, 63, 16), (129, 64, 17), (300, 44, 64),
                                             (257, 5, 65), (640, 33, 128), (148 * 128 + 1, 44, 5), (50000, 44, 8)])
def test_predictions_equal_the_layered_pass(rows, n_in, n_out):
    import torch
    net = _net(n_in, n_out, rows + n_out)
    g = torch.Generator(device="cuda").manual_seed(rows)
    X = torch.rand((rows, n_in), device="cuda", generator=g) * 2 - 1
    want = _layered(net, X)
    assert torch.equal(net.predict_device(X), want)
    assert np.array_equal(net.predict(X.cpu().numpy(), batch=1000), want.cpu().numpy())
    # rows of a wider matrix, and double-precision rows
    wide = torch.full((rows, n_in + 3), float("nan"), device="cuda")
    wide[:, 1:1 + n_in] = X
    assert torch.equal(net.predict_device(wide[:, 1:1 + n_in]), want)
    assert torch.equal(net.predict_device(X.double()), want)


@pytest.mark.parametrize("rows,n_in,n_out", [(1, 44, 5), (128, 10, 3), (129, 64, 17), (1000, 44, 5), (2048, 7, 64),
                                             (513, 44, 65), (700, 12, 128), (4096, 44, 5)])
def test_gradients_equal_the_layered_pass(rows, n_in, n_out):
    import torch
    net = _net(n_in, n_out, rows)
    rng = np.random.Generator(np.random.PCG64(rows))
    X = rng.uniform(-1, 1, size=(rows, n_in)).astype(np.float32)
    T = rng.normal(size=(rows, n_out)).astype(np.float32)
    mask = (rng.uniform(size=T.shape) > 0.3).astype(np.float32)
    mask[0, 0] = 1
    loss, dW, db = _layered(net, *(torch.tensor(v, device="cuda") for v in (X, T, mask)))
    T[mask == 0] = np.nan  # undefined targets are masked
    got, gW, gb = net.gradients(X, T, mask)
    assert abs(got - loss) <= 1e-5 * abs(loss)
    for i in range(4):
        assert torch.equal(gW[i], dW[i]) and torch.equal(gb[i], db[i]), i


@pytest.mark.parametrize("rows", [9000, 20000])
def test_gradients_of_large_batches(rows):
    """Longer row ranges per unit: float32 sums of the same products in
    another order."""
    import torch
    net = _net(44, 5, 1)
    rng = np.random.Generator(np.random.PCG64(rows))
    X = rng.uniform(-1, 1, size=(rows, 44)).astype(np.float32)
    T = rng.normal(size=(rows, 5)).astype(np.float32)
    mask = np.ones_like(T)
    loss, dW, db = _layered(net, *(torch.tensor(v, device="cuda") for v in (X, T, mask)))
    got, gW, gb = net.gradients(X, T, mask)
    assert abs(got - loss) <= 1e-5 * abs(loss)
    for i in range(4):
        assert torch.equal(gb[i], db[i])
        assert (gW[i] - dW[i]).norm() <= 1e-5 * dW[i].norm()


@pytest.mark.parametrize("rows,nets", [(1, 1), (130, 3), (20000, 4), (300, 64), (300, 65)])
def test_ranking_equals_the_separate_kernels(rows, nets):
    """The fused ranking against encode, layered networks, ensemble sum and
    score; 65 networks take the path of more than one launch."""
    import math

    import torch
    from dense_b200 import search as S
    from dense_b200.surrogate import IN_PAD
    idx = S.active_params()
    some = [_net(len(idx), 5, s) for s in range(min(nets, 4))]
    many = [some[i % len(some)] for i in range(nets)]
    sur = S.Surrogate(many, mu=[3.3, 3.9, 0.2, 0.0, 0.0], sd=[0.4, 0.8, 0.3, 1.0, 1.0])
    P = S.draw_candidates(rows, 7)
    k = some[0].k
    Pd = torch.tensor(P, device="cuda")
    Xb = torch.empty((rows, IN_PAD), dtype=torch.bfloat16, device="cuda")
    k.encode(Pd, torch.tensor(idx.astype(np.int32), device="cuda"), torch.tensor(S.template()[idx], device="cuda"),
             math.log(S.SPREAD), Xb)
    x = Xb[:, :len(idx)].float()
    ys = [_layered(n, x).contiguous() for n in some]
    acc = torch.empty((rows, 5), device="cuda")
    for i in range(nets):
        k.ensemble_accumulate(ys[i % len(some)], rows, 5, acc, i == 0)
    want = torch.empty(rows, dtype=torch.float64, device="cuda")
    k.score(acc, nets, sur.mu, sur.sd, S.REGION_WEIGHT, S.TARGET_PERIOD, S.PERIOD_TOL, S.AMP_MIN, S.AMP_RAMP, want)
    assert np.array_equal(S.score_candidates(sur, P), want.cpu().numpy())


def test_empty_inputs_and_refusals():
    import torch
    net = _net(44, 5, 2)
    assert net.predict_device(torch.zeros((0, 44), device="cuda")).shape == (0, 5)
    assert net.predict(np.zeros((0, 44), np.float32)).shape == (0, 5)
    with pytest.raises(RuntimeError):
        net.predict_device(torch.zeros((3, 43), device="cuda"))


@pytest.mark.parametrize("n_out", [5, 64, 65, 128])
@pytest.mark.parametrize("rows", [4097, 4224, 4225, 4353, 5000])
def test_gradients_around_the_last_cluster(rows, n_out):
    """One cluster of CTAs a tile up to as many as the GPU holds, one CTA a
    tile above: bias gradients bit for bit, weight gradients as sums of the
    same products in another order (float32, 1e-5)."""
    import torch
    net = _net(44, n_out, 1)
    rng = np.random.Generator(np.random.PCG64(rows))
    X = rng.uniform(-1, 1, size=(rows, 44)).astype(np.float32)
    T = rng.normal(size=(rows, n_out)).astype(np.float32)
    mask = (rng.uniform(size=T.shape) > 0.3).astype(np.float32)
    loss, dW, db = _layered(net, *(torch.tensor(v, device="cuda") for v in (X, T, mask)))
    got, gW, gb = net.gradients(X, T, mask)
    assert abs(got - loss) <= 1e-5 * abs(loss)
    for i in range(4):
        assert torch.equal(gb[i], db[i])
        assert (gW[i] - dW[i]).norm() <= 1e-5 * dW[i].norm()


@pytest.mark.parametrize("rows", [300, 6000])
def test_steps_in_a_captured_graph(rows):
    """Pass and finish of two steps, replayed: the weights of the same steps
    launched one by one."""
    import torch
    rng = np.random.Generator(np.random.PCG64(rows))
    f = lambda x: torch.tensor(x.astype(np.float32), device="cuda")  # noqa: E731
    X, T = f(rng.uniform(-1, 1, size=(rows, 44))), f(rng.normal(size=(rows, 5)))
    mask = torch.ones_like(T)
    hyper = f(np.array([[1e-3, 0.9, 0.999, 1e-8, 1 - 0.9 ** t, 1 - 0.999 ** t, 1.0 / rows, 0.0] for t in (1, 2)]))
    got = []
    for graph in (False, True):
        net = _net(44, 5, 3)
        work, loss = net._work(rows), torch.zeros(1, device="cuda")
        idx = torch.arange(rows, dtype=torch.int32, device="cuda").repeat(2)
        net._pack(backward=True)
        run = lambda: net.k.train_epoch(X, T, mask, idx, hyper, loss, work, net)  # noqa: E731
        if graph:
            held = [t.clone() for t in net.W + net.b]
            run()  # a first launch of each kernel
            for t, h in zip(net.W + net.b, held):
                t.copy_(h)
            for t in net.mW + net.vW + net.mb + net.vb:
                t.zero_()
            net._pack(backward=True)
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                run()
            g.replay()
        else:
            run()
        net.k.check()
        got.append([t.clone() for t in net.W + net.b])
    for a, b in zip(*got):
        assert torch.equal(a, b)
