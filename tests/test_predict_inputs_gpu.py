"""predict_device on inputs of other types and layouts than float32 rows: the
values of the float32 rows, and copies of `batch` rows at a time only."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _net_and_rows(rows, n_in=40):
    import torch
    from dense_b200.surrogate import MLP
    X = np.random.Generator(np.random.PCG64(1)).uniform(-1, 1, size=(rows, n_in)).astype(np.float32)
    return MLP(n_in, 5, seed=3), torch.from_numpy(X).cuda()


@pytest.mark.parametrize("batch", [1, 100, 65536])
@pytest.mark.parametrize("form", ["double", "half", "transposed", "wide", "one_row", "broadcast", "host"])
def test_forms(form, batch):
    import torch
    net, X = _net_and_rows(1 if form == "one_row" else 257)
    wide = torch.zeros((X.shape[0], 64), device="cuda")
    wide[:, 7:47] = X
    got, want = {
        "double": (X.double(), X),
        "half": (X.half(), X.half().float()),
        "transposed": (X.t().contiguous().t(), X),
        "wide": (wide[:, 7:47], X),
        # a row whose stride is no leading dimension
        "one_row": (torch.as_strided(X, (1, 40), (2 ** 33, 1)), X),
        "broadcast": (X[:, :1], X[:, :1].expand(257, 40).contiguous()),
        "host": (X.cpu(), X),
    }[form]
    # (float64 and float16 inputs are rounded to BF16 once, as the kernel does)
    assert torch.equal(net.predict_device(got, batch=batch), net.predict_device(want.to(torch.bfloat16).float()
                                                                               if form in ("double", "half") else want))


def test_conversions_take_a_batch_of_memory():
    import torch
    net, X = _net_and_rows(1 << 19)
    D = X.double()
    net.predict_device(D[:1000])
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = net.predict_device(D, batch=4096)
    peak = torch.cuda.max_memory_allocated() - before
    assert peak < out.numel() * 4 + 4 * 4096 * 40 * 4 + (4 << 20)
    assert torch.equal(out, net.predict_device(X.to(torch.bfloat16).float()))
