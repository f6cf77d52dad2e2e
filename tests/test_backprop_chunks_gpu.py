"""Gradients of many samples, where a chunk (mlp_backprop_kernel) has more than one set of 32 of them, against
the mean over parts that have one set per chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PART = 16000  # 500 sets: one per chunk, of at most 608


def _terms(torch, p, x, y):
    """Mean absolute value of every parameter's terms, in 64 bits."""
    p = torch.from_numpy(p.astype(np.float64)).cuda()
    at, w = 0, []
    for shape in ((64, 16), (64,), (64, 64), (64,), (3, 64), (3,)):
        k = int(np.prod(shape))
        w.append(p[at:at + k].view(shape))
        at += k
    x = (x.double() - p[at:at + 16]) / p[at + 16:at + 32]
    h1 = torch.relu(x @ w[0].t() + w[1])
    h2 = torch.relu(h1 @ w[2].t() + w[3])
    d3 = torch.softmax(h2 @ w[4].t() + w[5], 1) - torch.nn.functional.one_hot(y.long(), 3)
    d2 = (d3 @ w[4]) * (h2 > 0)
    d1 = (d2 @ w[2]) * (h1 > 0)
    out = []
    for d, a in ((d1, x), (d2, h1), (d3, h2)):
        out += [(d.abs().t() @ a.abs()).reshape(-1), d.abs().sum(0)]
    return (torch.cat(out) / len(x)).cpu().numpy()


@pytest.mark.parametrize("count", [19456, 19457, 20001, 38912, 38913, 50000])
def test_against_parts(lagpu, ctx_fast, count):
    """The samples' deltas are the same numbers either way, only the order of their sums differs: chains of
    up to 96 terms per thread, 76 chunks and 8 partial sums here, 32, 63 and 8 in the parts, in FP32, so
    within 300 * 2^-24 of the terms' mean absolute value (the mean of the parts is taken in 64 bits)."""
    torch = pytest.importorskip("torch")
    mlp = lagpu.Mlp(ctx_fast, 3)
    p = mlp.get_params()
    g = torch.Generator(device="cuda").manual_seed(count)
    x = torch.randn((count, 16), generator=g, device="cuda")
    y = torch.randint(0, 3, (count,), generator=g, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    got, loss = mlp.gradients(x.data_ptr(), y.data_ptr(), count)
    want, total = np.zeros(len(got)), 0.0
    for s in range(0, count, PART):
        k = min(PART, count - s)
        part, l = mlp.gradients(x[s:s + k].data_ptr(), y[s:s + k].data_ptr(), k)
        want += part.astype(np.float64) * k / count
        total += l * k / count
    mlp.free()
    # 2 % for terms that 64 bits see otherwise (a unit at its kink)
    assert np.all(np.abs(got - want) <= 300 * 2.0 ** -24 * (1.02 * _terms(torch, p, x, y) + 1e-12))
    assert abs(loss - total) <= 1e-6 * abs(total)
